// Device kernels of the FP64 path: cell binning and sort, SA-SPH boundary
// data, continuity and momentum pair passes, leapfrog, EoS and time step.
//
// Compiled with --fmad=false: every FP64 expression below is evaluated in
// the reference's left-to-right order without contraction, like the
// gfortran -O2 x86-64 build of the reference (src/Makefile:124), so the
// pair sums reproduce the reference's rounding.
#include <cstdint>
#include <cfloat>
#include "../../include/sphera_b200.h"
#include "sph_internal.cuh"
#include "sph_launch.h"

namespace sph {

// BoundIntegralTab2D (SA_SPH_module.f90:29-54), filled by the host with the
// single-precision roundings of the table's default-REAL literals.
__constant__ double c_bit2d[22][6];

namespace {

constexpr double kMaxPositive = 3.4e+38;       // max_positive_number
constexpr double kPigreco = 3.14159265358979e0;
constexpr double kKernelConst2D = 0.454728408833987e0;
constexpr double kDeltaXBit = 0.1;

// --------------------------------------------------------------------------
// small helpers
// --------------------------------------------------------------------------

// A launch made by launch_next may be set up while the last blocks of the one
// before it in its stream still run, and waits here, before it reads anything,
// until that one has finished and its writes are visible.  After an ordinary
// launch this returns at once.
__device__ __forceinline__ void chain_wait() {
  cudaGridDependencySynchronize();
}

__device__ __forceinline__ void load_sim(SimDev& dst, const SimDev* src, int sim, int& cur) {
  if (cur == sim) return;
  __syncthreads();
  const unsigned long long* s = reinterpret_cast<const unsigned long long*>(src + sim);
  unsigned long long* d = reinterpret_cast<unsigned long long*>(&dst);
  constexpr int n = sizeof(SimDev) / 8;
  for (int i = threadIdx.x; i < n; i += blockDim.x) d[i] = s[i];
  cur = sim;
  __syncthreads();
}

// ParticleCellNumber.f90:52-62 + CellNumber.f90:53-59: 1-based (i,j,k),
// false if outside the grid.
// a / b rounded to nearest, bit for bit what the IEEE division a / b gives,
// from y = RN(1/b) (a constant's reciprocal formed on the host, or
// __drcp_rn(b) once for a divisor that several divisions share).  The
// method is Markstein's (P. Markstein, IBM J. Res. Dev. 34(1), 1990; the
// theorem in Muller et al., Handbook of Floating-Point Arithmetic, on
// division with a fused multiply-add): if y is within half an ulp of 1/b
// and q within one ulp of a/b, the remainder r = a - b q is exact and
// RN(q + r y) = RN(a/b).  q0 = RN(a y) can be up to 1.5 ulp off, so one
// correction first brings it within half an ulp plus O(2^-105) relative
// (q1), and the second is the theorem's step.  A zero remainder means the
// current q is the exact quotient and is kept as it is (so a zero a keeps
// its sign, which q + 0 y would lose).  Domain: a, b finite, b != 0, and no
// quotient or remainder in the subnormal range -- true of every caller
// (lengths, densities and smoothing lengths of a physical state).
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  const double q0 = __dmul_rn(a, y);
  const double r0 = __fma_rn(-b, q0, a);
  const double q1 = r0 == 0.0 ? q0 : __fma_rn(r0, y, q0);
  const double r1 = __fma_rn(-b, q1, a);
  return r1 == 0.0 ? q1 : __fma_rn(r1, y, q1);
}

// div_rn without the two selections: the same quotient wherever it is not
// zero (a zero remainder adds a zero, which changes no nonzero number), and
// for a zero dividend a zero whose sign is the IEEE one except that -0 over
// a positive divisor gives +0.  For operands that cannot be -0 and for
// quotients whose zeros only ever meet a sum that started at +0.  The two
// compares are FP64 instructions: without them a pair of the FP64 momentum
// pass is 10 of its 202 FP64 instructions shorter, one of the matrix pass 30
// of about 230.
__device__ __forceinline__ double div_rn_unsigned0(double a, double b, double y) {
  const double q0 = __dmul_rn(a, y);
  const double q1 = __fma_rn(__fma_rn(-b, q0, a), y, q0);
  return __fma_rn(__fma_rn(-b, q1, a), y, q1);
}

// q >= 1 and q >= 2 for q >= 0, from its upper word (integer instructions).
// A NaN is at or beyond both: for pair terms that are multiplied by the
// separation (or hold the velocities it became NaN from) and are NaN anyway.
// A range test against it cost the FP64 step 0.2 to 0.6% (3D, from 256,000 particles).
__device__ __forceinline__ bool at_least_one(double q) { return __double2hiint(q) >= 0x3ff00000; }
__device__ __forceinline__ bool at_least_two(double q) { return __double2hiint(q) >= 0x40000000; }

__device__ __forceinline__ bool particle_cell(const SimDev& s, double x, double y, double z, int& i, int& j,
                                              int& k) {
  double ci = ceil(div_rn_unsigned0(x - s.extr_lo[0], s.dcd[0], s.rcp_dcd[0])) - (double)s.ioff;   // exact: whole numbers
  double ck = ceil(div_rn_unsigned0(z - s.extr_lo[2], s.dcd[2], s.rcp_dcd[2]));
  double cj = (s.dim == 3) ? ceil(div_rn_unsigned0(y - s.extr_lo[1], s.dcd[1], s.rcp_dcd[1])) : 1.0;
  if (!(ci >= 1.0 && ci <= (double)s.ncd[0] && cj >= 1.0 && cj <= (double)s.ncd[1] && ck >= 1.0 &&
        ck <= (double)s.ncd[2]))
    return false;
  i = (int)ci;
  j = (int)cj;
  k = (int)ck;
  return true;
}

// FP32 offset of a particle from the origin of its cell; w holds the cell's
// k index as a float (exact: k < 2^24), so cell differences are FP32
// subtractions, exact, with no integer-to-float conversion in the pair loops.
__device__ __forceinline__ float4 screening_copy(const SimDev& s, const double4& x, bool inside, int i, int j, int k) {
  if (!inside) return make_float4(0.f, 0.f, 0.f, -8.0f);
  double ox = s.extr_lo[0] + s.dcd[0] * (i + s.ioff - 1);
  double oy = (s.dim == 3) ? s.extr_lo[1] + s.dcd[1] * (j - 1) : 0.0;
  double oz = s.extr_lo[2] + s.dcd[2] * (k - 1);
  return make_float4((float)(x.x - ox), (float)(x.y - oy), (float)(x.z - oz), (float)k);
}

// Contiguous slot range of neighbour column r (reference order: y, then x).
template <int DIM>
__device__ __forceinline__ void neighbour_run(const SimDev& s, const int* __restrict__ cell_start, int ci, int cj,
                                              int ck, int r, int& b, int& e) {
  int jr = (DIM == 3) ? cj - 1 + r / 3 : cj;
  int ir = ci - 1 + ((DIM == 3) ? r % 3 : r);
  b = 0;
  e = 0;
  if (ir < 1 || ir > s.ncd[0] || jr < 1 || jr > s.ncd[1]) return;
  int klo = ck > 1 ? ck - 1 : 1;
  int khi = ck < s.ncd[2] ? ck + 1 : s.ncd[2];
  int base = s.cell_off + ((jr - 1) * s.ncd[0] + (ir - 1)) * s.ncd[2];
  b = __ldg(cell_start + base + klo - 1);
  e = __ldg(cell_start + base + khi);
}

// Kernel values of CalcVarLength.f90:242-269 for an accepted pair.
__device__ __forceinline__ void kernel_values(const SimDev& s, double rijtemp2, double& PK1, double& PK2,
                                              double& PK3) {
  double rijtemp = sqrt(rijtemp2);
  double rij_su_h = div_rn_unsigned0(rijtemp, s.h, s.rcp_h);
  double rij_su_h_quad = div_rn_unsigned0(rijtemp2, s.squareh, s.rcp_squareh);
  double denom = 1.0 / (rijtemp + s.eta);
  PK1 = 0.0;
  PK2 = 0.0;
  PK3 = 0.0;
  if (at_least_two(rij_su_h)) return;
  double gradmod = -(2.0 * rij_su_h) + 1.5 * rij_su_h_quad;
  double gradmodwacl = -12.0 - 3.0 * rij_su_h_quad + 12.0 * rij_su_h;
  if (at_least_one(rij_su_h)) gradmod = -gradmod + rij_su_h_quad - 2.0;
  gradmod = gradmod * s.ke_coef;
  gradmodwacl = gradmodwacl * s.kacl_coef;
  PK1 = gradmod * denom;
  PK2 = PK1 / (rijtemp2 + s.eta2);
  PK3 = gradmodwacl * denom;
}

__device__ __forceinline__ void set_status(SimDyn* d, int code) { atomicCAS(&d->status, 0, code); }

__device__ __forceinline__ double warp_min(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ int warp_max(int v) {
  for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Adds two per-thread counts of the block to counters[0..1] (one atomic per
// block and counter).
__device__ __forceinline__ void block_count2(unsigned long long* counters, int a, int c) {
  unsigned long long sa = (unsigned long long)a, sc = (unsigned long long)c;
  for (int o = 16; o > 0; o >>= 1) {
    sa += __shfl_xor_sync(0xffffffffu, sa, o);
    sc += __shfl_xor_sync(0xffffffffu, sc, o);
  }
  if ((threadIdx.x & 31) == 0 && (sa | sc)) {
    atomicAdd(counters, sa);
    atomicAdd(counters + 1, sc);
  }
}

// InterpolateTable.f90:58-82 on columns 1..4.
__device__ __forceinline__ void interpolate_table(const SimDev& s, double xval, double* iv) {
  double deltaX = s.ktdelta;
  double xval0 = s.kerneltab[0][0];
  int nr0 = (int)div_rn(xval - xval0, deltaX, s.rcp_ktdelta);
  if (nr0 <= 0) {
    for (int c = 0; c < 4; ++c) iv[c] = s.kerneltab[0][c + 1];
  } else if (nr0 >= kKtRows) {
    for (int c = 0; c < 4; ++c) iv[c] = s.kerneltab[kKtRows][c + 1];
  } else {
    double csi = div_rn(xval - s.kerneltab[nr0][0], deltaX, s.rcp_ktdelta);
    for (int c = 0; c < 4; ++c)
      iv[c] = s.kerneltab[nr0][c + 1] + csi * (s.kerneltab[nr0 + 1][c + 1] - s.kerneltab[nr0][c + 1]);
  }
}

// LocalNormalCoordinates.f90:59-87 + IsPointInternal.f90:54-72.
__device__ __forceinline__ bool point_internal(const FaceDev& f, double px, double py) {
  double c0 = (f.AA[0] + f.BB[0] * px + f.CC[0] * py) * f.usu_due_area;
  double c1 = (f.AA[1] + f.BB[1] * px + f.CC[1] * py) * f.usu_due_area;
  if (f.fkod == 2) return !(c0 < 0.0 || c0 > 1.0 || c1 < 0.0 || c1 > 1.0);
  if (f.fkod == 1) {
    double c2 = 1.0 - (c0 + c1);
    return !(c0 < 0.0 || c0 > 1.0 || c1 < 0.0 || c1 > 1.0 || c2 < 0.0 || c2 > 1.0);
  }
  return false;
}

// w.f90:48-57
__device__ __forceinline__ double w_kernel(double r, double h, double coef) {
  double s = r / h, q;
  if (s <= 1.0) q = 0.666666667 + s * s * (s * 0.5 - 1.0);
  else if (s >= 2.0) q = 0.0;
  else {
    double dms = 2.0 - s;
    q = dms * dms * dms / 6.0;
  }
  return q * coef;
}

// WIntegr.f90:57-74
__device__ __forceinline__ double w_integr(double ri, double hh) {
  double ro = ri / hh;
  if (0.0 <= ro && ro < 1.0) {
    double ro2 = ro * ro, ro3 = ro2 * ro;
    double W1 = (0.5 + -0.375 * ro2 + 0.15 * ro3) * ro2;
    return kKernelConst2D * (0.35 - W1);
  } else if (1.0 <= ro && ro < 2.0) {
    double q1 = 2.0 - ro, q2 = q1 * q1, q4 = q2 * q2;
    double W2 = (-0.125 + 0.05 * q1) * q4;
    return -kKernelConst2D * W2;
  }
  return 0.0;
}

// J2Wro2.f90:50-63
__device__ __forceinline__ double j2_wro2(double ro) {
  const double a1 = 0.00833333333333333, a2 = 0.26666666666666667;
  double ro2 = ro * ro, ro3 = ro2 * ro;
  if (0.0 <= ro && ro < 1.0) return kKernelConst2D * (0.25 - (a1 * (40.0 - 36.0 * ro2 + 15.0 * ro3) * ro3));
  if (1.0 <= ro && ro < 2.0)
    return kKernelConst2D * (a2 - (a1 * (80.0 - 90.0 * ro + 36.0 * ro2 - 5.0 * ro3) * ro3));
  return 0.0;
}

// InterpolateBoundaryIntegrals2D.f90:61-69
__device__ __forceinline__ void interp_bit2d(int ncols, const int* col, double xx, double* func) {
  if (xx < c_bit2d[0][0]) xx = c_bit2d[0][0];
  int ii = (int)((xx - c_bit2d[0][0]) / kDeltaXBit) + 1;
  if (ii > 21) ii = 21;  // the table ends at 2.001; deltai < 2 on this path
  double xi = c_bit2d[ii - 1][0];
  for (int nc = 0; nc < ncols; ++nc) {
    double fi = c_bit2d[ii - 1][col[nc]];
    double fip1 = c_bit2d[ii][col[nc]];
    func[nc] = fi + (fip1 - fi) * (xx - xi) / kDeltaXBit;
  }
}

}  // namespace

// ==========================================================================
// Sorting (OrdGrid1 replacement)
// ==========================================================================

// Copies the sorted state into the scratch record the sort consumes.
__global__ void k_stage(DevBatch b) {
  __shared__ SimDev s;
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count) continue;
    const Particles& P = b.P;
    double4 x = P.X[p];
    double4 v = P.V[p];
    double2 rp = P.RP[p];
    P.X2[p] = x;
    P.V2[p] = make_double4(v.x, v.y, v.z, rp.x);
    P.P2[p] = rp.y;
    P.I2[p] = P.I[p];
    P.L2[p] = P.L[p];
  }
}

constexpr int kScanThreads = 1024;
constexpr int kScanPer = 4;
constexpr int kScanChunk = kScanThreads * kScanPer;
constexpr int kBinChunks = 8;            // chunks around a block's first that k_bin gathers
constexpr int kMostOwnSums = 16384;      // chunks (67 10^6 cells) up to which k_scan's blocks add up the sums before them

// Cell key of every slot + atomic histogram, and the histogram's sums over
// chunks of kScanChunk cells that the scan starts from.  KeyKind::Sort bins the
// scratch record by the z-fastest layout key; KeyKind::Reference bins the
// sorted state by CellNumber.f90's numbering for the grid dump.
template <KeyKind KIND>
__global__ void k_bin(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  __shared__ int first_chunk, chunk_sum[kBinChunks];
  int cur = -1;
  const Particles& P = b.P;
  const int lane = threadIdx.x & 31;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    const bool valid = threadIdx.x < tl.count;
    int p = tl.start + threadIdx.x;
    int key = -1;
    if (valid) {
      SimDyn* dyn = b.dyn + tl.sim;
      int nag = dyn->nag;
      key = s.cell_off + s.ncells;  // removal bin
      if (p < s.p_off + nag) {
        double4 x = (KIND == KeyKind::Sort) ? P.X2[p] : P.X[p];
        int i, j, k;
        if (particle_cell(s, x.x, x.y, x.z, i, j, k)) {
          key = s.cell_off + ((KIND == KeyKind::Sort) ? cell_key_local(s, i, j, k)
                                                       : ((k - 1) * s.ncd[1] + (j - 1)) * s.ncd[0] + (i - 1));
        } else if (KIND == KeyKind::Sort) {
          atomicAdd(&dyn->n_out, 1);
          P.out_flag[s.p_off + P.I2[p] - 1] = 1;
        }
      }
      P.key[p] = key;
    }
    // the lanes of a warp that bin into one cell (the last sort's order
    // keeps most of a warp in one or two) take their slots with one atomic;
    // a slot only has to be unique within its cell (the placement is ranked
    // by caller index afterwards)
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    int base = 0;
    if (valid && lane == leader) base = atomicAdd(P.cell_count + key, __popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (valid) P.slot[p] = base + __popc(peers & ((1u << lane) - 1u));
    // the chunk sums of the scan, gathered over the block (its particles
    // lie in one chunk or a few): a global addition per warp met the others
    // on the same few addresses and cost 14 us at 864,000 particles
    const int chunk = valid ? key / kScanChunk : -1;
    if (threadIdx.x == 0) first_chunk = chunk;
    if (threadIdx.x < kBinChunks) chunk_sum[threadIdx.x] = 0;
    __syncthreads();
    const unsigned same = __match_any_sync(0xffffffffu, chunk);
    if (valid && lane == __ffs(same) - 1) {
      const unsigned c = (unsigned)(chunk - first_chunk + kBinChunks / 2);
      if (c < (unsigned)kBinChunks) atomicAdd(chunk_sum + c, __popc(same));
      else atomicAdd(b.scan_block_sums + chunk, __popc(same));
    }
    __syncthreads();
    if (threadIdx.x < kBinChunks && chunk_sum[threadIdx.x] != 0)
      atomicAdd(b.scan_block_sums + first_chunk - kBinChunks / 2 + threadIdx.x, chunk_sum[threadIdx.x]);
    __syncthreads();
  }
}

// OrdGrid1.f90:58-82: particles out of the grid are removed by moving the
// last particle into their place, in increasing particle index.  Replayed
// exactly (one thread per simulation, only when a removal happened).
__device__ void replay_removals(const DevBatch& b, int sim) {
  SimDyn* d = b.dyn + sim;
  if (d->n_out == 0) return;
  const SimDev& s = b.sims[sim];
  uint8_t* out = b.P.out_flag + s.p_off - 1;   // 1-based by caller index
  int* cur_of = b.P.cur_of + s.p_off - 1;
  int* remap = b.P.id_remap + s.p_off - 1;
  int n0 = d->nag;
  int n = n0;
  for (int id = 1; id <= n0; ++id) { cur_of[id] = id; remap[id] = 0; }
  int npi = 0;
  while (n > 0 && npi < n) {
    npi = npi + 1;
    if (out[npi]) {
      out[npi] = out[n];
      cur_of[npi] = cur_of[n];
      n = n - 1;
      npi = npi - 1;
    }
  }
  for (int id = 1; id <= n; ++id) remap[cur_of[id]] = id;
  for (int id = 1; id <= n0; ++id) out[id] = 0;
  d->removed_total += n0 - n;
  d->nag = n;
  d->warnings |= SPH_WARN_PARTICLES_REMOVED;
}

// Exclusive scan of v over the block, and its total.
__device__ __forceinline__ int block_excl_scan(int v, int* warp_sums, int& total) {
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int nw = blockDim.x >> 5;
    int ws = lane < nw ? warp_sums[lane] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, ws, o);
      if (lane >= o) ws += y;
    }
    if (lane < nw) warp_sums[lane] = ws;
  }
  __syncthreads();
  int base = wid > 0 ? warp_sums[wid - 1] : 0;
  total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return base + x - v;
}

// Exclusive scan of the cell histogram, clearing it: block c < nb handles
// one chunk of kScanChunk cells, starting from the sum of the chunk sums
// before it (k_bin added those up).  The blocks past the chunks replay the
// removals, one simulation each: both need the finished binning and
// neither needs the other, so one launch holds what were four (chunk sums,
// their scan, the scan, the removals).  These launches are latency alone:
// at 5,000 particles the sort took 35 us in eight launches.
//
// summed: the chunk sums have been made prefix sums already (k_scan_sums).
// Each block adding up all sums before its own is nothing for a few thousand
// chunks and grows with their square (a sort in 151 10^6 cells 885 us so and 816
// with prefix sums, in 302 10^6 1955 and 1591).
__global__ void __launch_bounds__(kScanThreads) k_scan(DevBatch b, int n, int nb, int* cell_start, int removals,
                                                       int summed) {
  chain_wait();
  if (blockIdx.x >= nb) {
    const int sim = blockIdx.x - nb;
    if (removals && threadIdx.x == 0 && sim < b.nsims) replay_removals(b, sim);
    return;
  }
  __shared__ int ws[32];
  __shared__ int before;
  int* cnt = b.P.cell_count;
  const int base = blockIdx.x * kScanChunk + threadIdx.x * kScanPer;
  int vals[kScanPer];
  int v = 0;
  for (int q = 0; q < kScanPer; ++q) {
    vals[q] = (base + q < n) ? cnt[base + q] : 0;
    v += vals[q];
  }
  int prev = 0;
  if (summed) prev = threadIdx.x == 0 ? b.scan_block_sums[blockIdx.x] : 0;
  else
    for (int c = threadIdx.x; c < (int)blockIdx.x; c += kScanThreads) prev += b.scan_block_sums[c];
  if (threadIdx.x == 0) before = 0;
  __syncthreads();
  prev = __reduce_add_sync(0xffffffffu, prev);
  if ((threadIdx.x & 31) == 0 && prev) atomicAdd(&before, prev);
  int total;
  int ex = block_excl_scan(v, ws, total);
  ex += before;
  for (int q = 0; q < kScanPer; ++q) {
    if (base + q < n) {
      cell_start[base + q] = ex;
      cnt[base + q] = 0;
    }
    ex += vals[q];
    if (base + q == n - 1) cell_start[n] = ex;
  }
}

// The chunk sums in place of their exclusive prefix sums, by one block, for the
// grids of very many chunks (kMostOwnSums).
__global__ void __launch_bounds__(kScanThreads) k_scan_sums(int* sums, int nb) {
  __shared__ int ws[32];
  int carry = 0;
  for (int c0 = 0; c0 < nb; c0 += kScanThreads) {
    const int c = c0 + threadIdx.x;
    const int v = c < nb ? sums[c] : 0;
    int total;
    const int ex = block_excl_scan(v, ws, total);
    if (c < nb) sums[c] = carry + ex;
    carry += total;
  }
}

__device__ __forceinline__ void reset_boundary_counters(const DevBatch& b, int sim) {
  b.dyn[sim].ncbf_max = 0;
  b.dyn[sim].bdt_sim_used = 0;
  if (sim == 0) b.dyn[b.nsims].bdt_used = 0;
}

// Unstable placement by cell (the atomic slot), remembering the source.
// Also clears the scan's chunk sums for the next binning and, where the
// boundary pass follows, that pass's counters.
__global__ void k_place(DevBatch b, const int* __restrict__ cstart, int use_scratch_ids, int boundary_follows) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < b.scan_nblocks; c += gridDim.x * blockDim.x)
    b.scan_block_sums[c] = 0;
  if (boundary_follows)
    for (int sim = blockIdx.x * blockDim.x + threadIdx.x; sim < b.nsims; sim += gridDim.x * blockDim.x)
      reset_boundary_counters(b, sim);
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    if (threadIdx.x >= tl.count) continue;
    int p = tl.start + threadIdx.x;
    int key = P.key[p];
    int dst = cstart[key] + P.slot[p];
    int id = use_scratch_ids ? P.I2[p] : P.I[p];
    if (use_scratch_ids && b.dyn[tl.sim].n_out > 0 && id > 0) id = P.id_remap[s.p_off + id - 1];
    P.tmp_src[dst] = p;
    P.tmp_id[dst] = id;
    P.tmp_key[dst] = key;
  }
}

// Rank inside the cell by caller index (OrdGrid1.f90:100-105 stable
// scatter) and gather the scratch record into the sorted state.
// PART selects what is gathered: kPermuteAll everything (the step); the IC
// of an upload splits it in two so that the velocities, densities and
// pressures can still be on their way from the host while the lists and
// the boundary data are built from the sorted positions:
// kPermutePositions gathers x, m, the caller index and the laminar flag and
// keeps each slot's destination in P.slot (free once k_place has run);
// kPermuteRest gathers the rest through it.
constexpr int kPermuteAll = 0, kPermutePositions = 1, kPermuteRest = 2;

template <int PART>
__global__ void __launch_bounds__(kBlock) k_rank_permute(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  if (PART != kPermuteRest)   // the out-of-grid count, for the next binning
    for (int sim = blockIdx.x * blockDim.x + threadIdx.x; sim < b.nsims; sim += gridDim.x * blockDim.x)
      b.dyn[sim].n_out = 0;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    if (threadIdx.x >= tl.count) continue;
    int d = tl.start + threadIdx.x;
    int fin = d;
    if (PART == kPermuteRest) {
      fin = P.slot[d];
    } else {
      int key = P.tmp_key[d];
      int myid = P.tmp_id[d];
      if (key != s.cell_off + s.ncells) {
        int cs = P.cell_start[key], ce = P.cell_start[key + 1];
        int rank = 0;
        for (int q = cs; q < ce; ++q) rank += (P.tmp_id[q] < myid) ? 1 : 0;
        fin = cs + rank;
      }
      P.I[fin] = myid;
      if (PART == kPermutePositions) P.slot[d] = fin;
    }
    int src = P.tmp_src[d];
    double4 x = P.X2[src];
    if (PART != kPermuteRest) {
      P.X[fin] = x;
      int ic, jc, kc;
      const bool inside = particle_cell(s, x.x, x.y, x.z, ic, jc, kc);
      P.XF[fin] = screening_copy(s, x, inside, ic, jc, kc);
      P.L[fin] = P.L2[src];
    }
    if (PART != kPermutePositions) {
      double4 v = P.V2[src];
      double vol = x.w / v.w;
      double pr = P.P2[src];
      P.V[fin] = make_double4(v.x, v.y, v.z, vol);
      P.RP[fin] = make_double2(v.w, pr);
      // the FP32 records only where a pass reads them: the FP64 form has no
      // use for them, and RF is the smoothing passes' alone (40 of the 225
      // bytes this launch moves per particle, 16 in the FP32c form)
      if (b.fp32c) {
        P.VF[fin] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)vol);
        const float prr = (float)(pr / (v.w * v.w));
        P.RM[fin] = make_float2((float)v.w, prr);
        if (b.smooths) P.RF[fin] = make_float4((float)v.w, prr, (float)x.w, 0.f);
      }
    }
  }
}

// NPartOrd of the reference numbering (verification only).
__global__ void k_rank_reference(DevBatch b, const int* __restrict__ cstart, int* npartord) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    if (threadIdx.x >= tl.count) continue;
    int d = tl.start + threadIdx.x;
    int key = P.tmp_key[d];
    if (key == s.cell_off + s.ncells) continue;
    int myid = P.tmp_id[d];
    int cs = cstart[key], ce = cstart[key + 1];
    int rank = 0;
    for (int q = cs; q < ce; ++q) rank += (P.tmp_id[q] < myid) ? 1 : 0;
    npartord[cs + rank - s.p_off] = myid;
  }
}

// ==========================================================================
// SA-SPH boundary data (ComputeBoundaryDataTab_3D / _2D)
// ==========================================================================

// ComputeBoundaryVolumeIntegrals_P0.f90:81-155 for one (particle, face).
// The point-in-face test of one face held in registers (the same arithmetic
// as point_internal).
struct FaceTest {
  double a0, a1, b0, b1, c0, c1, u;
  int fkod;
  __device__ __forceinline__ void load(const FaceDev& f) {
    a0 = f.AA[0];
    a1 = f.AA[1];
    b0 = f.BB[0];
    b1 = f.BB[1];
    c0 = f.CC[0];
    c1 = f.CC[1];
    u = f.usu_due_area;
    fkod = f.fkod;
  }
  __device__ __forceinline__ bool inside(double px, double py) const {
    double k0 = (a0 + b0 * px + c0 * py) * u;
    double k1 = (a1 + b1 * px + c1 * py) * u;
    if (fkod == 2) return !(k0 < 0.0 || k0 > 1.0 || k1 < 0.0 || k1 > 1.0);
    if (fkod == 1) {
      double k2 = 1.0 - (k0 + k1);
      return !(k0 < 0.0 || k0 > 1.0 || k1 < 0.0 || k1 > 1.0 || k2 < 0.0 || k2 > 1.0);
    }
    return false;
  }
};

// The hemisphere table as the quadrature reads it.  coef(q, l, .) are the
// factors of point q in the three sums of lane l: (1, 1, r2 r2), (r0, r1,
// r2), (r0 r0, r0 r1, r0 r2) and (r1 r1, r1 r2, r2 r2).
struct BitTable {
  const double (*xy)[2];      // [256] x, y of the points
  const double (*ring)[2];    // [8] z and weight of a ring's points (the same for all of them)
  const double (*cf)[12];     // [256] the factors, lane by lane
  __device__ __forceinline__ double x(int q) const { return xy[q][0]; }
  __device__ __forceinline__ double y(int q) const { return xy[q][1]; }
  __device__ __forceinline__ double z(int r) const { return ring[r][0]; }
  __device__ __forceinline__ double da(int r) const { return ring[r][1]; }
  __device__ __forceinline__ void coef(int q, int l, double* c) const {
    for (int k = 0; k < 3; ++k) c[k] = cf[q][3 * l + k];
  }
};

// ComputeBoundaryVolumeIntegrals_P0.f90:81-155 for one (particle, face) by
// four neighbouring lanes.  Its 256 points add to twelve sums one after the
// other; each lane keeps three of them (l = 0: IntWdV, IntdWrm1dV,
// IntGWZrm1dV; 1: G; 2: R00, R01, R02; 3: R11, R12, R22), every sum in the
// reference's order.  The points' tests are shared out over the lanes, and
// left out for a face that the whole projected hemisphere lies inside
// (`whole`, with a margin far above the test's rounding): most entries of a
// wall that is large against 2h.  The chain of one entry is what bounds
// this pass: by one lane (12 sums, 256 tests and the products of the
// factors, which come from the table here) it took 65 us at 13,500
// particles and 143 us at 864,000.
__device__ __forceinline__ void face_integrals(const SimDev& s, const BitTable& bit, const FaceDev& f,
                                               const double* locx, int l, double* sum) {
  FaceTest ft;
  ft.load(f);
  sum[0] = sum[1] = sum[2] = 0.0;
  const double L0 = locx[0], L1 = locx[1];
  double L2 = locx[2];
  if (L2 < 0.0) return;
  if (L2 < s.zpmin) L2 = s.zpmin;
  const unsigned group = 0xfu << (threadIdx.x & 28);
  bool whole;
  {
    // a projected point lies within 2h of (L0, L1); the test's coordinates
    // are linear in it
    const double R = s.doubleh * 1.000001, u = fabs(ft.u);
    const double k0 = (ft.a0 + ft.b0 * L0 + ft.c0 * L1) * ft.u, k1 = (ft.a1 + ft.b1 * L0 + ft.c1 * L1) * ft.u;
    const double d0 = (fabs(ft.b0) + fabs(ft.c0)) * R * u, d1 = (fabs(ft.b1) + fabs(ft.c1)) * R * u;
    const double m = 1.0e-12 + 1.0e-12 * u * (fabs(ft.a0) + fabs(ft.a1) + (fabs(ft.b0) + fabs(ft.b1)) * (fabs(L0) + R) +
                                              (fabs(ft.c0) + fabs(ft.c1)) * (fabs(L1) + R));
    whole = k0 - d0 > m && k0 + d0 < 1.0 - m && k1 - d1 > m && k1 + d1 < 1.0 - m;
    if (ft.fkod == 1) {
      const double k2 = 1.0 - (k0 + k1), d2 = d0 + d1, m2 = 2.0 * m;
      whole = whole && k2 - d2 > m2 && k2 + d2 < 1.0 - m2;
    }
  }
  double J0 = 0.0, J1 = 0.0, J2 = 0.0, J3 = 0.0;   // the kernel-table values of the last refresh
  double Ja = 0.0, Jb = 0.0;                       // this lane's: of its first sum, of the other two
  double robpre = 2.1;
  for (int ring = 0; ring < 8; ++ring) {
    const double zp = bit.z(ring);
    const double lpj2 = L2 + zp;
    if (!(lpj2 <= 0.0)) continue;       // the whole ring lies above the face plane
    const double tsegnato = L2 / (L2 - lpj2);
    const int q0 = ring * 32;
    auto project = [&](int q, double& px0, double& px1) {
      const double lpj0 = L0 + bit.x(q), lpj1 = L1 + bit.y(q);
      px0 = L0 + (lpj0 - L0) * tsegnato;
      px1 = L1 + (lpj1 - L1) * tsegnato;
    };
    unsigned in = 0xffffffffu;
    if (!whole) {
      in = 0u;
      for (int k = 0; k < 8; ++k) {
        const int q = 4 * k + l;
        double px0, px1;
        project(q0 + q, px0, px1);
        if (ft.inside(px0, px1)) in |= 1u << q;
      }
      in |= __shfl_xor_sync(group, in, 1);
      in |= __shfl_xor_sync(group, in, 2);
    }
    if (in == 0u) continue;
    // |rob - robpre| > 1e-3 at point q: new table values
    auto refresh = [&](int q) {
      double px0, px1;
      project(q, px0, px1);
      const double d0 = px0 - L0, d1 = px1 - L1, d2 = 0.0 - L2;
      const double dist = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
      const double rob = div_rn_unsigned0(dist, s.h, s.rcp_h);
      const double gap = fabs(rob - robpre);
      if (gap > 1.0e-3) {
        double iv[4];
        interpolate_table(s, rob, iv);
        const double da = bit.da(ring);
        J0 = iv[0] * da;
        J1 = iv[1] * da;
        J2 = iv[2] * da;
        J3 = iv[3] * da;
        Ja = l == 0 ? J0 : (l == 1 ? J2 : J3);
        Jb = l == 0 ? J1 : (l == 1 ? J2 : J3);
        robpre = rob;
      }
      return gap;
    };
    auto add = [&](int q) {
      double c[3];
      bit.coef(q, l, c);
      sum[0] = sum[0] + c[0] * Ja;
      sum[1] = sum[1] + c[1] * Jb;
      sum[2] = sum[2] + c[2] * Jb;
    };
    // The points of a ring share their polar angle, so their distances to
    // the particle differ by rounding only (s.ring_skip bounds that far
    // below 1e-6 in rob).  After the ring's first inside point the
    // refresh test |rob - robpre| > 1e-3 is therefore false for every
    // later point -- unless the first point missed the threshold by less
    // than 1e-6, when the ring is tested point by point.  Skipping the
    // test skips its distance, square root and division.
    const double gap = refresh(q0 + __ffs(in) - 1);
    const bool test_all = !s.ring_skip || (!(gap > 1.0e-3) && gap > 1.0e-3 - 1.0e-6);
    if (test_all) {
      bool first = true;
      for (int q = 0; q < 32; ++q) {
        if (!((in >> q) & 1u)) continue;
        if (!first) refresh(q0 + q);
        first = false;
        add(q0 + q);
      }
    } else if (in == 0xffffffffu) {
#pragma unroll 8
      for (int q = 0; q < 32; ++q) add(q0 + q);
    } else {
      for (int q = 0; q < 32; ++q)
        if ((in >> q) & 1u) add(q0 + q);
    }
  }
  if (l == 0 && L2 == s.zpmin) sum[0] = point_internal(f, L0, L1) ? 0.5 : 0.0;
}

// Room for n boundary entries of each lane's particle (one simulation to a
// warp): the first entry, or -1 where n is 0 or there is none.  Each
// simulation draws on its own part of the pool, so one that overflows fails
// alone and the others' entries are unaffected; what is left of the part when
// a particle's entries don't fit is marked (face 0), so that every entry
// below the count is one of this pass.  One addition per warp and counter: a
// lane's own met all the others at one address (72 us for the
// 864,000-particle dam break's face search).
__device__ __forceinline__ int claim_entries(const SimDev& s, const DevBatch& b, SimDyn* dyn, int n) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (!__any_sync(FULL, n > 0)) return -1;
  int inc = n, base = 0;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(FULL, inc, o);
    if (lane >= o) inc += u;
  }
  if (lane == 31) base = atomicAdd(&dyn->bdt_sim_used, inc);
  base = __shfl_sync(FULL, base, 31);
  const int first = base + inc - n;
  if (n > 0 && base + inc > s.bdt_quota) {
    set_status(dyn, SPH_ERR_BDT_OVERFLOW);
    for (int k = first; k < s.bdt_quota; ++k) b.P.bdt[s.bdt_off + k].clobonum = 0;
    n = 0;
  }
  const int taken = __reduce_add_sync(FULL, n);
  if (lane == 31 && taken > 0) atomicAdd(&b.dyn[b.nsims].bdt_used, taken);   // of all simulations (diagnostics)
  return n > 0 ? s.bdt_off + first : -1;
}

// ComputeBoundaryDataTab_3D.f90:67-105 with FindCloseBoundaryFaces3D.f90:79-188:
// a particle's close faces, in the order the 27 cells around its cell name
// them, become entries of the boundary table (their integrals are a pass of
// their own).  The host has merged the 27 cells' face lists into one list
// per cell, each face at its first place: a particle reads that list instead
// of 27.
__global__ void __launch_bounds__(kBlock) k_boundary3d(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    const int p = tl.start + threadIdx.x;
    const bool slot = threadIdx.x < tl.count;
    SimDyn* dyn = b.dyn + tl.sim;
    int clob[kMaxLocalFaces];
    double pin[kMaxLocalFaces];
    int ncbf = 0;
    double4 x = make_double4(0.0, 0.0, 0.0, 0.0);
    int ic, jc, kc;
    if (slot && p < s.p_off + dyn->nag && s.nfaces > 0) x = P.X[p];
    if (slot && p < s.p_off + dyn->nag && s.nfaces > 0 && particle_cell(s, x.x, x.y, x.z, ic, jc, kc)) {
      const int gk = s.cell_off + cell_key_local(s, ic, jc, kc);
      const int nf = b.cf_count[gk];
      const int fs = nf > 0 ? b.cf_start[gk] : 0;
      bool overflow = false;
      for (int q = 0; q < nf; ++q) {
        const int fid = b.cf_list[fs + q];
        const FaceDev& f = b.faces[s.face_off + fid - 1];
        double pn = 0.0;
        pn = pn + f.T[0][2] * (x.x - f.GXref[0]);
        pn = pn + f.T[1][2] * (x.y - f.GXref[1]);
        pn = pn + f.T[2][2] * (x.z - f.GXref[2]);
        if (pn >= 0.0 && pn < s.doubleh) {
          if (ncbf >= s.maxcb || ncbf >= kMaxLocalFaces) {
            overflow = true;
          } else {
            clob[ncbf] = fid;
            pin[ncbf] = pn;
          }
          ncbf++;
        }
      }
      if (overflow) {
        set_status(dyn, SPH_ERR_CLOSE_FACES);
        ncbf = 0;
      }
    }
    const int gbase = claim_entries(s, b, dyn, ncbf);
    if (gbase < 0) ncbf = 0;
    if (slot) P.bdt_count[p] = ncbf;
    const int most = warp_max(ncbf);
    if ((threadIdx.x & 31) == 0 && most > 0) atomicMax(&dyn->ncbf_max, most);
    if (ncbf == 0) continue;
    P.bdt_start[p] = gbase;
    for (int u = 0; u < ncbf; ++u) {
      const FaceDev& f = b.faces[s.face_off + clob[u] - 1];
      double locx[3];
      for (int sdi = 0; sdi < 2; ++sdi) {
        double acc = 0.0;
        acc = acc + f.T[0][sdi] * (x.x - f.GXref[0]);
        acc = acc + f.T[1][sdi] * (x.y - f.GXref[1]);
        acc = acc + f.T[2][sdi] * (x.z - f.GXref[2]);
        locx[sdi] = acc;
      }
      locx[2] = pin[u];
      BdtEntry& e = P.bdt[gbase + u];
      e.loc[0] = locx[0];
      e.loc[1] = locx[1];
      e.loc[2] = locx[2];
      e.clobonum = clob[u];
    }
  }
}

// The integrals of entry e by its four lanes.
__device__ __forceinline__ void boundary_entry(const SimDev& s, const BitTable& bit, const DevBatch& b, BdtEntry& e,
                                               int l) {
  if (e.clobonum == 0) return;
  const double locx[3] = {e.loc[0], e.loc[1], e.loc[2]};
  double sum[3];
  face_integrals(s, bit, b.faces[s.face_off + e.clobonum - 1], locx, l, sum);
  if (l == 0) {
    e.bi[0] = 0.0;
    e.bi[1] = sum[0];
    e.bi[2] = sum[1];
    e.bi[6] = sum[2];
    e.bi[7] = 0.0;
  } else if (l == 1) {
    for (int k = 0; k < 3; ++k) e.bi[3 + k] = sum[k];
  } else if (l == 2) {
    e.ig[0] = sum[0];
    e.ig[1] = e.ig[3] = sum[1];
    e.ig[2] = e.ig[6] = sum[2];
  } else {
    e.ig[4] = sum[0];
    e.ig[5] = e.ig[7] = sum[1];
    e.ig[8] = sum[2];
  }
}

// ComputeBoundaryVolumeIntegrals_P0.f90:81-155 for every entry the find
// pass allocated, four lanes to a (particle, face): the quadrature costs are
// balanced across the GPU whatever the particles' distribution over tiles.
// A block works on chunks of 32 entries of one simulation, whose constants and
// hemisphere table it holds in shared memory; the chunks of 128 simulations at a
// time are numbered through, one simulation after the other.  (Entries of a
// pool that the members share as they come mix in a chunk, and those of another
// member than the table's read theirs from global memory: 300 members of 500
// particles 806 us, 20 of 13,500 457; with a part of the pool each 372 and 201.)
__global__ void __launch_bounds__(128) k_boundary3d_integrals(DevBatch b) {
  chain_wait();
  constexpr int PER = 32, GROUP = 128;
  __shared__ SimDev ssim;
  __shared__ double sxy[kBitRows][2];
  __shared__ double sring[8][2];
  __shared__ double scf[kBitRows][12];
  __shared__ int ends[GROUP], part[GROUP / 32];   // chunks up to the end of each simulation of the group
  int loaded = -1;
  const int l = threadIdx.x & 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto entries = [&](int sim) { return min(b.dyn[sim].bdt_sim_used, b.sims[sim].bdt_quota); };
  int before = 0, next = blockIdx.x;               // chunks of the groups so far; this block's next one
  for (int s0 = 0; s0 < b.nsims; s0 += GROUP) {
    int end = s0 + (int)threadIdx.x < b.nsims ? (entries(s0 + threadIdx.x) + PER - 1) / PER : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    __syncthreads();                               // the last group's ends are no longer read
    if (lane == 31) part[warp] = end;
    __syncthreads();
    end += before;
    for (int w = 0; w < warp; ++w) end += part[w];
    ends[threadIdx.x] = end;
    __syncthreads();
    for (; next < ends[GROUP - 1]; next += gridDim.x) {
      int k = 0;                                   // the first simulation that ends past the chunk
      for (int step = GROUP / 2; step > 0; step >>= 1)
        if (ends[k + step - 1] <= next) k += step;
      const int sim = s0 + k, chunk = next - (k > 0 ? ends[k - 1] : before);
      if (sim != loaded) {
        load_sim(ssim, b.sims, sim, loaded);
        const double* src = b.bit + (size_t)sim * kBitRows * 7;
        for (int q = threadIdx.x; q < kBitRows; q += blockDim.x) {
          const double* row = src + 7 * q;
          const double r0 = row[4], r1 = row[5], r2 = row[6];
          sxy[q][0] = row[0];
          sxy[q][1] = row[1];
          if ((q & 31) == 0) {
            sring[q >> 5][0] = row[2];
            sring[q >> 5][1] = row[3];
          }
          const double c[12] = {1.0, 1.0, r2 * r2, r0, r1, r2, r0 * r0, r0 * r1, r0 * r2, r1 * r1, r1 * r2, r2 * r2};
          for (int j = 0; j < 12; ++j) scf[q][j] = c[j];
        }
        __syncthreads();
      }
      const int idx = chunk * PER + (threadIdx.x >> 2);
      if (idx < entries(sim)) boundary_entry(ssim, BitTable{sxy, sring, scf}, b, b.P.bdt[ssim.bdt_off + idx], l);
    }
    before = ends[GROUP - 1];
  }
}

// The integrals of a particle close to two sides (a corner), both entries
// at a time by one warp: lanes 0-15 the first, 16-31 the second.  Each of
// the three quadratures has at most 10 abscissae (an arc of at most pi in
// steps of about pi / 10; a chord of at most 4 h in steps of about h / 2), so
// a lane forms one term of each -- its abscissa by the reference's repeated
// addition -- and the terms are summed in the reference's order.  One lane
// doing all of a corner's sines, cosines, tangents and arc tangents in
// sequence took 37 us at 5,000 particles, the longest launch of a 2D step.
__device__ __forceinline__ void corner_integrals2d(const SimDev& s, const SideDev* __restrict__ sd, SimDyn* dyn,
                                                   const int* ib, const double* ix, const double* iy,
                                                   BdtEntry* out) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, i = lane & 15, c = lane >> 4;
  const double px = c ? ix[1] : ix[0], py = c ? iy[1] : iy[0];
  const int isi = c ? ib[1] : ib[0];
  // the half's terms 0..n-1 added to acc in order
  auto add_terms = [&](double acc, double term, int n) {
    for (int k = 0; k < 16; ++k) {
      const double v = __shfl_sync(FULL, term, k, 16);
      if (k < n) acc = acc + v;
    }
    return acc;
  };
  auto sub_terms = [&](double acc, double term, int n) {
    for (int k = 0; k < 16; ++k) {
      const double v = __shfl_sync(FULL, term, k, 16);
      if (k < n) acc = acc - v;
    }
    return acc;
  };
  // FindBoundaryIntersection2D.f90:61-92
  const double minlen = 0.01 * s.h;
  const double ypi = py < 0.0 ? 0.0 : py;
  const double halfchord = sqrt(s.square_doubleh - ypi * ypi);
  const double XA = px - halfchord, XB = px + halfchord;
  double xpmin = 0.0;
  if (XA > xpmin) xpmin = XA;
  double xpmax = sd[isi - 1].length;
  if (XB < xpmax) xpmax = XB;
  double interlen = xpmax - xpmin;
  if (interlen <= minlen) interlen = 0.0;
  const bool cut = interlen > 0.0;
  // ComputeSurfaceIntegral_WdS2D.f90:57-83
  int ndiv = 0;
  double term = 0.0;
  if (cut) {
    const double dsrif = s.h / 2;
    const double ypiq = ypi * ypi;
    ndiv = (int)(interlen / dsrif + 0.5);
    if (ndiv < 2) ndiv = 2;
    const double deltas = interlen / ndiv;
    double xpip = xpmin - 0.5 * deltas;
    for (int k = 0; k <= i; ++k) xpip = xpip + deltas;
    const double dxpip = xpip - px;
    const double ris = sqrt(dxpip * dxpip + ypiq);
    term = w_kernel(ris, s.h, s.coefke) * deltas;
  }
  const double IntWdS = add_terms(0.0, term, ndiv);
  // BoundaryVolumeIntegrals2D.f90
  const double dalfarif = kPigreco / 10;
  const double yplimite = 0.05 * s.h;
  const double ypb = py < yplimite ? yplimite : py;
  double alfaA = 0.0, Intalfa = 0.0, t0 = 0.0, t1 = 0.0, t2 = 0.0;
  ndiv = 0;
  if (cut) {
    alfaA = atan2(xpmin - px, ypb);
    Intalfa = atan2(xpmax - px, ypb) - alfaA;
    ndiv = (int)(Intalfa / dalfarif + 0.5);
    if (ndiv < 1) ndiv = 1;
    const double dalfa = Intalfa / ndiv;
    double alfa_k = alfaA - 0.5 * dalfa;
    for (int k = 0; k <= i; ++k) alfa_k = alfa_k + dalfa;
    if (i < ndiv) {
      const double sa = sin(alfa_k), ca = cos(alfa_k);
      const double rb = ypb / ca;
      const double rob = div_rn(rb, s.h, s.rcp_h);
      const double mult = s.h * j2_wro2(rob) * dalfa;
      t0 = sa * mult;
      t1 = ca * mult;
      t2 = w_integr(rb, s.h) * dalfa;
    }
  }
  const double D0 = add_terms(0.0, t0, ndiv);
  const double D1 = sub_terms(0.0, t1, ndiv);
  double IntWdV = add_terms(0.0, t2, ndiv);
  if (cut && ypb == yplimite) IntWdV = 0.5;
  // ComputeVolumeIntegral_WdV2D.f90; at py >= yplimite (so ypb = py) its arc
  // is the one above
  term = 0.0;
  const bool arc = cut && py >= yplimite;
  ndiv = 0;
  if (arc) {
    ndiv = (int)(Intalfa / dalfarif + 0.5);
    if (ndiv < 2) ndiv = 2;
    const double dalfa = Intalfa / ndiv;
    double alfa = alfaA - 0.5 * dalfa;
    for (int k = 0; k <= i; ++k) alfa = alfa + dalfa;
    if (i < ndiv) {
      const double ta = tan(alfa);
      const double ris = py * sqrt(1.0 + ta * ta);
      term = w_integr(ris, s.h) * dalfa;
    }
  }
  double IntWdV1 = add_terms(0.0, term, ndiv);
  if (cut && !arc) {
    const double ypj = c ? iy[0] : iy[1];   // the other side
    if (ypj <= yplimite) {
      double angle = 0.0;
      if (sd[ib[0] - 1].previous_side == ib[1]) angle = sd[ib[0] - 1].angle;
      else if (sd[ib[1] - 1].previous_side == ib[0]) angle = sd[ib[1] - 1].angle;
      else set_status(dyn, 804);
      IntWdV1 = 0.5 * (angle + kPigreco) / (2.0 * kPigreco);
    } else {
      IntWdV1 = (xpmin >= px && px <= xpmax) ? 0.5 : 0.0;
    }
  }
  if (i != 0) return;
  double func[3];
  const int col[3] = {3, 4, 5};
  interp_bit2d(3, col, py / s.h, func);
  BdtEntry e;
  for (int q = 0; q < 9; ++q) e.ig[q] = 0.0;
  e.clobonum = isi;
  e.pad = 0;
  e.loc[0] = px;
  e.loc[1] = py;
  e.loc[2] = 0.0;
  e.bi[0] = IntWdS;
  e.bi[1] = IntWdV;
  e.bi[2] = IntWdV1;
  e.bi[3] = D0;
  e.bi[4] = D1;
  e.bi[5] = func[0] / s.squareh;
  e.bi[6] = func[1] / s.squareh;
  e.bi[7] = func[2] / s.squareh;
  out[c] = e;
}

// ComputeBoundaryDataTab_2D.f90:70-157 with FindCloseBoundarySides2D,
// SelectCloseBoundarySides2D, FindBoundaryIntersection2D,
// ComputeSurfaceIntegral_WdS2D, BoundaryVolumeIntegrals2D,
// ComputeVolumeIntegral_WdV2D and InterpolateBoundaryIntegrals2D.  A
// particle close to one side finishes its entry itself; the corner particles
// of the block (neighbours in the cell order) are then shared out over its
// warps (corner_integrals2d).
//
// It runs beside the list pass, whose blocks of 64 threads leave room for one
// of their own kind at a time: a block of 256 found a place late, and the pass,
// hidden before those small blocks came, cost its own time again (256 columns,
// 4.48 10^6 particles in FP32c: 2.305 ms a step with blocks of 256, 2.261 of 128,
// 2.253 of 64; 2.307 with lists in blocks of 256 as well).  Few tiles want the
// corners shared over more warps, and the FP64 form, which has no pair sums
// beside the pass, more of them: T = 128 from 8 tiles an SM in FP32c (80,000
// particles: 76.6 us a step with 128, 75.3 with 256; 320,000: 179.1 and 180.3;
// 500,000: 263.1 and 268.1; 1.02 10^6: 479 and 484) and from 32 in FP64 (80,000:
// 120.0 and 117.1; 500,000: 418 and 411; 1.02 10^6: 773 and 769; 2.28 10^6 in 128
// columns: 1723 and 1743).
template <int T>
__global__ void __launch_bounds__(T) k_boundary2d(DevBatch b) {
  chain_wait();
  constexpr int PARTS = kBlock / T;   // a tile's parts
  __shared__ SimDev s;
  __shared__ int ncorner, corner_ib[T][2], corner_base[T];
  __shared__ double corner_xy[T][4];   // x of both entries, y of both
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles * PARTS; t += gridDim.x) {
    Tile tl = b.tiles[t / PARTS];
    load_sim(s, b.sims, tl.sim, cur);
    const int at = (t % PARTS) * T + threadIdx.x;
    const int p = tl.start + at;
    const bool slot = at < tl.count;
    SimDyn* dyn = b.dyn + tl.sim;
    if (slot) P.bdt_count[p] = 0;
    const bool on = slot && p < s.p_off + dyn->nag && s.nsides > 0;
    const SideDev* sd = b.sides + s.side_off;
    // SelectCloseBoundarySides2D: fixe / tapi sides in front of the particle
    int ib[kMaxCloseSides] = {0, 0, 0, 0};
    double ix[kMaxCloseSides] = {0.0, 0.0, 0.0, 0.0}, iy[kMaxCloseSides] = {0.0, 0.0, 0.0, 0.0};
    int nint = 0, gbase = 0;
    if (on) {
      double4 x = P.X[p];
      int clob[kMaxCloseSides];
      double lx[kMaxCloseSides], ly[kMaxCloseSides];
      int ncbs = 0;
      bool overflow = false;
      for (int isi = 1; isi <= s.nsides; ++isi) {
        const SideDev& S = sd[isi - 1];
        double P1P0 = x.x - S.v1[0], P1P1 = x.z - S.v1[1];
        double sidel = S.length;
        double xp = P1P0 * S.sss[0] + P1P1 * S.sss[1];
        double yp = P1P0 * S.nnn[0] + P1P1 * S.nnn[1];
        double xpmin = -s.doubleh, xpmax = sidel + s.doubleh;
        double ypmin = -s.doubleh, ypmax = s.doubleh;
        if ((xpmin < xp && xp < xpmax) && (ypmin < yp && yp < ypmax)) {
          double ypmx = 0.0, ypmn = 0.0;
          if (xp < 0.0) {
            ypmx = sqrt(s.square_doubleh - xp * xp);
            ypmn = -ypmx;
          } else if (xp <= sidel) {
            ypmx = ypmax;
            ypmn = ypmin;
          } else if (xp < xpmax) {
            double L = (sidel - xp) * (sidel - xp);
            ypmx = sqrt(s.square_doubleh - L);
            ypmn = -ypmx;
          }
          if (ypmn < yp && yp < ypmx) {
            if (ncbs >= kMaxCloseSides) {
              overflow = true;
            } else {
              clob[ncbs] = isi;
              lx[ncbs] = xp;
              ly[ncbs] = yp;
            }
            ncbs++;
          }
        }
      }
      if (overflow) {
        set_status(dyn, SPH_ERR_CLOSE_SIDES);
        ncbs = 0;
      }
      if (ncbs == 2) {
        if (sd[clob[0] - 1].previous_side == clob[1]) lx[1] = sd[clob[1] - 1].length - lx[1];
        else if (sd[clob[1] - 1].previous_side == clob[0]) lx[0] = sd[clob[0] - 1].length - lx[0];
      }
      for (int c = 0; c < ncbs; ++c)
        if (ly[c] > 0.0) {
          ib[nint] = clob[c];
          ix[nint] = lx[c];
          iy[nint] = ly[c];
          nint++;
        }
    }
    gbase = claim_entries(s, b, dyn, nint);
    if (gbase < 0) nint = 0;
    if (nint > 0) {
      P.bdt_count[p] = nint;
      P.bdt_start[p] = gbase;
    }
    if (nint == 1 || nint > 2) {
      for (int c = 0; c < nint; ++c) {
        BdtEntry e;
        for (int q = 0; q < 9; ++q) e.ig[q] = 0.0;
        for (int q = 0; q < 8; ++q) e.bi[q] = 0.0;
        e.clobonum = ib[c];
        e.pad = 0;
        e.loc[0] = ix[c];
        e.loc[1] = iy[c];
        e.loc[2] = 0.0;
        if (nint == 1) {
          double func[5];
          const int col[5] = {1, 2, 3, 4, 5};
          interp_bit2d(5, col, iy[c] / s.h, func);
          e.bi[0] = func[0] / s.h;
          e.bi[1] = func[1];
          e.bi[2] = func[1];
          e.bi[5] = func[2] / s.squareh;
          e.bi[6] = func[3] / s.squareh;
          e.bi[7] = func[4] / s.squareh;
        }
        P.bdt[gbase + c] = e;
      }
    }
    if (threadIdx.x == 0) ncorner = 0;
    __syncthreads();
    if (nint == 2) {
      const int c = atomicAdd(&ncorner, 1);
      corner_ib[c][0] = ib[0];
      corner_ib[c][1] = ib[1];
      corner_xy[c][0] = ix[0];
      corner_xy[c][1] = ix[1];
      corner_xy[c][2] = iy[0];
      corner_xy[c][3] = iy[1];
      corner_base[c] = gbase;
    }
    __syncthreads();
    for (int c = threadIdx.x >> 5; c < ncorner; c += T / 32)
      corner_integrals2d(s, sd, dyn, corner_ib[c], corner_xy[c], corner_xy[c] + 2, P.bdt + corner_base[c]);
    __syncthreads();
  }
}

// ==========================================================================
// Momentum: RHS_momentum_equation + inter_EqMoto + viscomon + viscomorris
// + AddBoundaryContributions_to_ME3D/2D + AddElasticBoundaryReaction_3D/2D,
// optionally fused with Leapfrog_momentum, velocity_smoothing_2 (TetaV=0),
// Leapfrog_trajectories and the CFL part of time_step_duration.
// ==========================================================================

// ---------------------------------------------------------------------------
// 1st-order consistency (input_any_t%C1_BE, %C1_divu; 3D).  The matrices are
// held as 9 doubles B(i,j) at 3 i + j, component-major over the slots.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void load_b(const double* __restrict__ src, int total, int p, double* B) {
  for (int k = 0; k < 9; ++k) B[k] = src[(size_t)k * total + p];
}

__device__ __forceinline__ void store_b(double* dst, int total, int p, const double* B) {
  for (int k = 0; k < 9; ++k) dst[(size_t)k * total + p] = B[k];
}

// Matrix_Inversion_3x3.f90:50-74 as B_ren_gradp_inversion.f90:58-74 and
// B_ren_divu_inversion.f90 use it: the inverse where |det| >= the
// threshold, else -I.
__device__ __forceinline__ void b_inversion(double* B, double thresh) {
  const double det = B[0] * B[4] * B[8] + B[3] * B[7] * B[2] + B[6] * B[1] * B[5] - B[0] * B[7] * B[5] -
                     B[6] * B[4] * B[2] - B[3] * B[1] * B[8];
  if (fabs(det) >= thresh) {
    double inv[9];
    inv[0] = B[4] * B[8] - B[5] * B[7];
    inv[1] = B[2] * B[7] - B[1] * B[8];
    inv[2] = B[1] * B[5] - B[2] * B[4];
    inv[3] = B[5] * B[6] - B[3] * B[8];
    inv[4] = B[0] * B[8] - B[2] * B[6];
    inv[5] = B[2] * B[3] - B[0] * B[5];
    inv[6] = B[3] * B[7] - B[4] * B[6];
    inv[7] = B[1] * B[6] - B[0] * B[7];
    inv[8] = B[0] * B[4] - B[1] * B[3];
    for (int k = 0; k < 9; ++k) B[k] = inv[k] / det;
  } else {
    for (int k = 0; k < 9; ++k) B[k] = 0.0;
    B[0] = B[4] = B[8] = -1.0;
  }
}

// v <- -(B v): MatrixProduct.f90 followed by the sign change of
// inter_EqMoto.f90:255-260, AddBoundaryContributions_to_ME3D.f90:320-325,
// SASPH_continuity.f90:126-140 and Continuity_Equation.f90:201-217.
__device__ __forceinline__ void b_renormalise(const double* B, double* v) {
  double a[3];
  for (int i = 0; i < 3; ++i) {
    double sum = 0.0;
    for (int k = 0; k < 3; ++k) sum = sum + B[3 * i + k] * v[k];
    a[i] = sum;
  }
  for (int i = 0; i < 3; ++i) v[i] = -a[i];
}

// The SA-SPH frontier's contribution T (IntGiWrRdV T^T) to the matrices,
// AddBoundaryContributions_to_ME3D.f90:172-187 and
// AddBoundaryContribution_to_CE3D.f90:93-112, added into B.
__device__ __forceinline__ void add_frontier_b(const FaceDev& f, const BdtEntry& e, double* B) {
  double m2[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double sum = 0.0;
      for (int k = 0; k < 3; ++k) sum = sum + e.ig[3 * i + k] * f.T[j][k];
      m2[3 * i + j] = sum;
    }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      double sum = 0.0;
      for (int k = 0; k < 3; ++k) sum = sum + f.T[i][k] * m2[3 * k + j];
      B[3 * i + j] = B[3 * i + j] + sum;
    }
}

// AddBoundaryContributions_to_ME3D.f90:105-336 (fixe/tapi, slip mode 1).
// C1: B is B_ren_gradp; on the first step (first) the frontiers add to it
// and it is inverted here, after the face loop; gradpt is renormalised.
template <bool C1 = false>
__device__ __forceinline__ void me_boundary3d(const SimDev& s, const DevBatch& b, int nb, int start, const double* vi, double rhoi,
                              double pres, int lam, const double* grav, double* tpres, double* tdiss, double* tvisc,
                              double* B = nullptr, bool first = false) {
  double ALEt[3] = {0, 0, 0}, gradpt[3] = {0, 0, 0}, VMon[3] = {0, 0, 0}, VShear[3] = {0, 0, 0};
  for (int u = 0; u < nb; ++u) {
    const BdtEntry& e = b.P.bdt[start + u];
    const FaceDev& f = b.faces[s.face_off + e.clobonum - 1];
    if (!(e.loc[2] > 0.0)) continue;
    double dvn = 0.0;
    for (int SD = 0; SD < 3; ++SD) {
      double dvij = 2.0 * (vi[SD] - f.velocity[SD]);
      dvn = dvn + f.T[SD][2] * dvij;
    }
    double gl[3];
    for (int SD = 0; SD < 3; ++SD) {
      double a = 0.0;
      for (int sdj = 0; sdj < 3; ++sdj) a = a + f.T[sdj][SD] * grav[sdj];
      gl[SD] = a;
    }
    double loc[3];
    for (int i = 0; i < 3; ++i) {
      double a = 0.0;
      for (int k = 0; k < 3; ++k) a = a + e.ig[3 * i + k] * gl[k];
      loc[i] = a;
    }
    for (int i = 0; i < 3; ++i) {
      double a = 0.0;
      for (int k = 0; k < 3; ++k) a = a + f.T[i][k] * loc[k];
      gradpt[i] = gradpt[i] + a;
    }
    double aloc[3];
    for (int k = 0; k < 3; ++k) aloc[k] = 2.0 * pres / rhoi * e.bi[3 + k];
    for (int i = 0; i < 3; ++i) {
      double a = 0.0;
      for (int k = 0; k < 3; ++k) a = a + f.T[i][k] * aloc[k];
      ALEt[i] = ALEt[i] + a;
    }
    if (C1 && first) add_frontier_b(f, e, B);
    double IntGWZrm1dV = e.bi[6];
    double IntdWrm1dV = e.bi[2];
    if (s.alfa_mon > 0.0) {
      double Monvisc = s.alfa_mon * s.celerita * s.h;
      double Mmult = -(Monvisc * dvn * IntGWZrm1dV);
      for (int d = 0; d < 3; ++d) VMon[d] = VMon[d] + Mmult * f.T[d][2];
    }
    double cinvisci = s.kin_visc;
    if (cinvisci > 0.0 && (lam == 1 || !f.laminar_no_slip_check)) {
      double cinviscmult = cinvisci * IntdWrm1dV * f.slip;
      for (int d = 0; d < 3; ++d) VShear[d] = VShear[d] + cinviscmult * (2.0 * (vi[d] - f.velocity[d]));
    }
  }
  if (C1) {
    if (first) b_inversion(B, s.invb_det_thresh);
    b_renormalise(B, gradpt);
  }
  for (int d = 0; d < 3; ++d) {
    tpres[d] = tpres[d] + ALEt[d] + gradpt[d];
    tdiss[d] = tdiss[d] - VMon[d];
    tvisc[d] = tvisc[d] + VShear[d];
  }
}

// AddBoundaryContributions_to_ME2D.f90:96-402 (fixe/tapi, slip mode 1).
__device__ __forceinline__ void me_boundary2d(const SimDev& s, const DevBatch& b, int nb, int start, const double* vi, double roi,
                              double pressi, int lam, const double* grav, double* tpres, double* tdiss, double* tvisc) {
  const double pibmink = 10.0;
  double ro0 = s.den0, distpimin = s.dx;
  double VMon[2] = {0, 0}, VShear[2] = {0, 0}, RG_sum[2] = {0, 0}, ALEt[2] = {0, 0};
  const double g2[2] = {grav[0], grav[2]};
  const double v2[2] = {vi[0], vi[2]};
  for (int u = 0; u < nb; ++u) {
    const BdtEntry& e = b.P.bdt[start + u];
    const SideDev& S = b.sides[s.side_off + e.clobonum - 1];
    double xpi = e.loc[0], ypi = e.loc[1];
    double IntWdS = e.bi[0], IntWdV = e.bi[2], IntWd1s0 = e.bi[5], IntWd3s0 = e.bi[6];
    double GravN = 0.0;
    for (int i = 0; i < 2; ++i) GravN = GravN + g2[i] * S.nnn[i];
    double sidevel[2] = {0.0, 0.0};
    if (S.zone_type == SPH_ZONE_TAPI) {
      sidevel[0] = S.velocity[0];
      sidevel[1] = S.velocity[2];
    }
    double Dvel0 = 2.0 * (v2[0] - sidevel[0]), Dvel1 = 2.0 * (v2[1] - sidevel[1]);
    double DvelN = Dvel0 * S.nnn[0] + Dvel1 * S.nnn[1];
    double distpi = fmax(ypi, distpimin);
    double pressib = pressi;
    double pressibmin = pibmink * ro0 * distpimin;
    if (DvelN <= 0.0 && pressib < pressibmin) pressib = pressibmin;
    double PressB = pressib - ro0 * GravN * distpi;
    double QiiIntWdS = IntWdS * (pressib + PressB) / roi;
    for (int i = 0; i < 2; ++i) {
      double RG = 0.0;
      for (int j = 0; j < 2; ++j) RG = RG + S.RN[i][j] * g2[j];
      RG = RG * IntWdV;
      RG_sum[i] = RG_sum[i] + RG;
    }
    ALEt[0] = ALEt[0] - S.nnn[0] * QiiIntWdS;
    ALEt[1] = ALEt[1] - S.nnn[1] * QiiIntWdS;
    if (xpi >= 0.0 && xpi <= S.length) {
      double Monvisc = s.alfa_mon * s.celerita * s.h;
      double TN = Monvisc * DvelN * IntWd3s0;
      double SVforce;
      if (lam == 1 || !S.laminar_no_slip_check) SVforce = 2.0 * s.kin_visc * S.slip * IntWd1s0;
      else SVforce = 0.0;
      for (int i = 0; i < 2; ++i) {
        VMon[i] = VMon[i] + TN * S.nnn[i];
        VShear[i] = VShear[i] + (2.0 * v2[i]) * SVforce;
      }
    }
  }
  const int acix[2] = {0, 2};
  for (int i = 0; i < 2; ++i) {
    tpres[acix[i]] = tpres[acix[i]] - RG_sum[i] - ALEt[i];
    tdiss[acix[i]] = tdiss[acix[i]] - VMon[i];
    tvisc[acix[i]] = tvisc[acix[i]] - VShear[i];
  }
}

// AddElasticBoundaryReaction_3D.f90:67-154 / _2D.f90:63-97; xi is
// pg%coord, vi pg%var (= pg%vel).
template <int DIM>
__device__ __forceinline__ void elastic_reaction(const SimDev& s, const DevBatch& b, int nb, int start, const double* xi,
                                                 const double* vi, double* R) {
  R[0] = R[1] = R[2] = 0.0;
  double zimin = 0.25 * s.dx;
  double celer02 = s.eps / s.den0;
  for (int u = 0; u < nb; ++u) {
    const BdtEntry& e = b.P.bdt[start + u];
    if (DIM == 3) {
      const FaceDev& f = b.faces[s.face_off + e.clobonum - 1];
      double zi = e.loc[2];
      if (zi < zimin && point_internal(f, e.loc[0], e.loc[1])) {
        double vin = 0.0;
        for (int sd = 0; sd < 3; ++sd) vin = vin + vi[sd] * f.T[sd][2];
        if (vin < 0.0) {
          double normreact = -(1.0 * celer02 * log((s.h + zi - zimin) / s.h) / s.h);
          for (int d = 0; d < 3; ++d) R[d] = R[d] + normreact * f.T[d][2];
        }
      }
    } else {
      const SideDev& S = b.sides[s.side_off + e.clobonum - 1];
      double xpi = e.loc[0], ypi = e.loc[1];
      if (ypi < zimin && xpi > 0.0 && xpi < S.length) {
        double vin = 0.0;
        vin = vin + vi[0] * S.nnn[0];
        vin = vin + vi[1] * 0.0;
        vin = vin + vi[2] * S.nnn[1];
        if (vin < 0.0) {
          double normreact = -(1.0 * celer02 * log((s.h + ypi - zimin) / s.h) / s.h);
          R[0] = R[0] + normreact * S.nnn[0];
          R[2] = R[2] + normreact * S.nnn[1];
        }
      }
    }
  }
  if (DIM == 3 && s.nedges > 0) {
    // Reaction from close convex edges (AddElasticBoundaryReaction_3D.f90:106-153).
    // ReaFace(icbf) -- the face term above applied its test to the entry --
    // is recomputed from the entry here.  An edge counts only when both of
    // its faces are close faces of the particle without a face reaction;
    // the reference leaves the routine at the first edge that fails this,
    // and so does this loop.
    auto rea_face = [&](const BdtEntry& e) {
      const FaceDev& f = b.faces[s.face_off + e.clobonum - 1];
      return e.loc[2] < zimin && point_internal(f, e.loc[0], e.loc[1]);
    };
    for (int ne = 0; ne < s.nedges; ++ne) {
      const EdgeDev& E = b.edges[s.edge_off + ne];
      int nclose = 0;
      for (int u = 0; u < nb; ++u) {
        const BdtEntry& e = b.P.bdt[start + u];
        if ((e.clobonum == E.face[0] || e.clobonum == E.face[1]) && !rea_face(e)) nclose++;
      }
      if (nclose != 2) break;
      double scaprod = 0.0;
      for (int sd = 0; sd < 3; ++sd) scaprod = scaprod + (xi[sd] - E.gx[sd]) * E.comp[sd];
      const double edgelen2 = E.length * E.length;
      const double tau = scaprod / edgelen2;
      if (tau >= 0.0 && tau <= 1.0) {
        double QP[3], edgedist2 = 0.0;
        for (int sd = 0; sd < 3; ++sd) QP[sd] = xi[sd] - (E.gx[sd] + E.comp[sd] * tau);
        for (int sd = 0; sd < 3; ++sd) edgedist2 = edgedist2 + QP[sd] * QP[sd];
        const double zi = sqrt(edgedist2);
        if (zi < zimin) {
          double cosdir[3], vin = 0.0;
          for (int sd = 0; sd < 3; ++sd) cosdir[sd] = QP[sd] / zi;
          for (int sd = 0; sd < 3; ++sd) vin = vin + vi[sd] * cosdir[sd];
          if (vin < 0.0) {
            const double normreact = -(1.0 * celer02 * log(zi / zimin) / zimin);
            for (int sd = 0; sd < 3; ++sd) R[sd] = R[sd] + normreact * cosdir[sd];
          }
        }
      }
    }
  }
}

// ==========================================================================
// Neighbour lists (the replacement of
// CalcVarLength.f90:133-269).  One pass after the sort stores, per particle,
// the slots of its accepted neighbours (the particle itself excluded, its
// acceptance still counted for the NMAXPARTJ cap) in the reference's
// visiting order: runs in (y, x) order, slots increasing inside a run.  Only
// 4-byte slot indices are kept, never kernel values or separations (the
// reference keeps 60 B per slot); every pass recomputes those.  The list of a
// step serves its continuity pass and the next step's momentum pass, which
// see the same positions.
//
// Layout: chunks of four entries (list_base4).  An entry is
// slot | (run << 28); the run gives the FP32 form the cell-origin difference
// of the pair.
//
// The scan is warp-cooperative: the lanes of a warp that share a (y, x) cell
// column (nearly always all of them, particles being sorted z-fastest) read
// the runs of their common window, drop what is far from all of them, and
// test what is left in lockstep, 32 candidates at a time from shared memory;
// each lane keeps the candidates of its own k-1..k+1 window, in the order of
// the runs, so its accepted sequence is exactly its reference order.
// ==========================================================================
constexpr int kSplitThreads = 128;   // threads of the four-lane FP64 pair passes
constexpr int kSlotBits = 28;
constexpr int kSlotMask = (1 << kSlotBits) - 1;

// Entries are stored as 16-byte chunks of 4: chunk c of particle p sits at
// int4 index ((p / 32) * cap4 + c) * 32 + p % 32, so a warp reading chunk c
// of its 32 particles reads 512 contiguous bytes.
__device__ __forceinline__ size_t list_base4(int p, int cap4) {
  return (size_t)(p >> 5) * (size_t)cap4 * 32 + (size_t)(p & 31);
}


// A warp's list region -- its chunks 0 .. ceil(nmax / 4) - 1, 512 B each
// and contiguous -- requested into L2 by one bulk prefetch from lane 0, so
// the chunk loads of the pair loop find it in L2 instead of waiting on HBM
// (the lists of a full-size step, 4 B per pair, do not stay in L2 between
// the pass that writes them and the passes that read them).  A hint only:
// 16-byte aligned address, a size in multiples of 16 bytes, no completion.
__device__ __forceinline__ void prefetch_list_l2(const int* nlist, int p, int cap4, int nmax) {
  if ((threadIdx.x & 31) != 0 || nmax <= 0) return;
  const int4* a = reinterpret_cast<const int4*>(nlist) + (size_t)(p >> 5) * (size_t)cap4 * 32;
  const unsigned bytes = (unsigned)((nmax + 3) >> 2) * 512u;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"(bytes) : "memory");
}

// A neighbour's 32-byte record in one 256-bit load (sm_100; the compiler
// splits a double4 into two 128-bit ones): half the gather instructions of
// the FP64 pair passes, and one L1 lookup per record instead of two.
__device__ __forceinline__ double4 load_record(const double4* p) {
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

// Sequential reader that loads chunk c + 1 while chunk c is consumed, so
// the list's HBM latency overlaps four pairs' work.
struct ListPrefetcher {
  const int4* base;
  int4 cur, nxt;
  int nchunks;
  __device__ __forceinline__ void init(const int* nlist, int p, int cap4, int cnt) {
    base = reinterpret_cast<const int4*>(nlist) + list_base4(p, cap4);
    nchunks = (cnt + 3) >> 2;
    nxt = nchunks > 0 ? __ldg(base) : make_int4(0, 0, 0, 0);
  }
  __device__ __forceinline__ int get(int k) {
    if ((k & 3) == 0) {
      cur = nxt;
      int c = (k >> 2) + 1;
      if (c < nchunks) nxt = __ldg(base + (size_t)c * 32);
    }
    int e = cur.x;
    cur.x = cur.y;
    cur.y = cur.z;
    cur.z = cur.w;
    return e;
  }
};

// r^2 <= (2h)^2 (CalcVarLength.f90:223-228) is decided on the FP32
// screening copies outside a band around (2h)^2 that the host derives from
// the copies' rounding bounds ([rr_lo, rr_hi]), and in FP64, exactly as the
// reference, inside it (one particle in 40 has such a candidate).  Candidates
// are staged in the frame of the group's lowest cell, f_j + D in x and y and
// (kj - kmin) dcd + f_j in z, so each difference costs one addition; the band
// covers that form's rounding for groups that span up to kMostSpan cells
// (sph_api.cu).

// Screens the staged tile of nt >= 1 candidates (negated x, y, z arrays) for
// one lane: bit 31 - u of the result is the sign of r^2 - mid of candidate u,
// and `near` falls to the least |r^2 - mid|, so that outside the band the
// sign is the test.  Candidates u, u + 1 share each paired FP32 instruction
// (__fadd2_rn, __fmul2_rn, __ffma2_rn), and one funnel shift moves a sign in.
// Entries past nt are staged far away and never hit.
template <int DIM>
__device__ __forceinline__ unsigned screen_tile(const float* nx, const float* ny, const float* nz, int nt, float ax,
                                                float ay, float zi, float mid, float& near) {
  const float2 ax2 = make_float2(ax, ax), ay2 = make_float2(ay, ay), zi2 = make_float2(zi, zi);
  const float2 nm2 = make_float2(-mid, -mid);
  unsigned m = 0u;
#pragma unroll
  for (int u0 = 0; u0 < 32; u0 += 8) {
    if (u0 >= nt) break;
#pragma unroll
    for (int c = 0; c < 8; c += 4) {
      const float4 X = *reinterpret_cast<const float4*>(nx + u0 + c);
      const float4 Z = *reinterpret_cast<const float4*>(nz + u0 + c);
      float2 ra = __fadd2_rn(ax2, make_float2(X.x, X.y));
      float2 rb = __fadd2_rn(ax2, make_float2(X.z, X.w));
      const float2 za = __fadd2_rn(zi2, make_float2(Z.x, Z.y));
      const float2 zb = __fadd2_rn(zi2, make_float2(Z.z, Z.w));
      ra = __fmul2_rn(ra, ra);
      rb = __fmul2_rn(rb, rb);
      if (DIM == 3) {
        const float4 Y = *reinterpret_cast<const float4*>(ny + u0 + c);
        const float2 ya = __fadd2_rn(ay2, make_float2(Y.x, Y.y));
        const float2 yb = __fadd2_rn(ay2, make_float2(Y.z, Y.w));
        ra = __ffma2_rn(ya, ya, ra);
        rb = __ffma2_rn(yb, yb, rb);
      }
      ra = __fadd2_rn(__ffma2_rn(za, za, ra), nm2);
      rb = __fadd2_rn(__ffma2_rn(zb, zb, rb), nm2);
      near = fminf(near, fminf(fabsf(ra.x), fabsf(ra.y)));
      near = fminf(near, fminf(fabsf(rb.x), fabsf(rb.y)));
      m = __funnelshift_l(__float_as_uint(ra.x), m, 1);
      m = __funnelshift_l(__float_as_uint(ra.y), m, 1);
      m = __funnelshift_l(__float_as_uint(rb.x), m, 1);
      m = __funnelshift_l(__float_as_uint(rb.y), m, 1);
    }
  }
  return m << (32 - ((nt + 7) & ~7));
}

// Run r of a cell's block: its candidates end before `end`, candidate c of
// the block is slot base + c, (dx, dy) the run's column origin in the cell's
// frame.
struct ListRun {
  int end, base;
  float dx, dy;
};

// The list of particle q, FP32 copy xq in cell (ci, cj, ck), by the whole
// warp: its own 27-cell block, 32 candidates at a time, the entries ranked by
// ballots and written one by one; the first NMAXPARTJ accepted are kept, the
// particle itself among them (CalcVarLength.f90:197-205), and trunc tells
// that candidates follow them.  For groups of few lanes, and for those whose
// common window is many times a particle's own.
template <int DIM>
__device__ __forceinline__ void list_by_ballots(const SimDev& s, const DevBatch& b, int q, const float4& xq, int ci,
                                                int cj, int ck, ListRun* runs, int& cnt, int& acc, int& cand,
                                                bool& trunc) {
  constexpr int NR = (DIM == 3) ? 9 : 3, UN = (DIM == 3) ? 4 : 2;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const Particles& P = b.P;
  const int cap = s.nmaxpartj;
  int nb = 0, ne = 0;
  if (lane < NR) neighbour_run<DIM>(s, P.cell_start, ci, cj, ck, lane, nb, ne);
  int inc = ne - nb;
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const int v = __shfl_up_sync(FULL, inc, o, 16);
    if ((lane & 15) >= o) inc += v;
  }
  __syncwarp();
  if (lane < NR) {
    const int rx = (DIM == 3) ? lane % 3 : lane;
    runs[lane] = ListRun{inc, nb - (inc - (ne - nb)), (float)(rx - 1) * s.dcdf[0],
                         (DIM == 3) ? (float)(lane / 3 - 1) * s.dcdf[1] : 0.f};
  }
  __syncwarp();
  const int W = __shfl_sync(FULL, inc, NR - 1);
  int* const list = b.nlist + 4 * list_base4(q, b.list_cap4);
  int total = 0, last = -1, r = 0;
  bool self_seen = false, self_kept = false;
  for (int g0 = 0; g0 < W; g0 += 32 * UN) {
    // UN candidates a lane, their loads in flight together
    int e[UN];
    float4 f[UN];
#pragma unroll
    for (int k = 0; k < UN; ++k) {
      const int c = g0 + 32 * k + lane;
      e[k] = -1;
      if (c < W) {
        while (c >= runs[r].end) ++r;
        e[k] = (runs[r].base + c) | (r << kSlotBits);
        f[k] = __ldg(P.XF + (runs[r].base + c));
      }
    }
#pragma unroll
    for (int k = 0; k < UN; ++k) {
      const int c0 = g0 + 32 * k;
      if (c0 >= W) break;
      bool hit = false, self = false;
      const int slot = e[k] & kSlotMask;
      if (e[k] != -1) {
        const int rk = (int)((unsigned)e[k] >> kSlotBits);
        const float d0 = xq.x - (f[k].x + runs[rk].dx), d1 = (DIM == 3) ? xq.y - (f[k].y + runs[rk].dy) : 0.f;
        const float d2 = xq.z - ((f[k].w - (float)ck) * s.dcdf[2] + f[k].z);
        const float rr = __fmaf_rn(d2, d2, __fmaf_rn(d1, d1, __fmul_rn(d0, d0)));
        hit = !(rr > s.rr_hi);
        if (hit && !(rr < s.rr_lo)) {
          const double4 xj = P.X[slot], xi = P.X[q];
          const double r0 = xi.x - xj.x, r1 = xi.y - xj.y, r2 = xi.z - xj.z;
          hit = !(r0 * r0 + r1 * r1 + r2 * r2 > s.square_doubleh);
        }
        self = hit && slot == q;
      }
      const unsigned m = __ballot_sync(FULL, hit), ms = __ballot_sync(FULL, self);
      const int rank = total + __popc(m & below);
      if (hit && !self && rank < cap) {
        const int pos = rank - ((self_seen || (ms & below)) ? 1 : 0);
        list[(size_t)(pos >> 2) * 128 + (pos & 3)] = e[k];
      }
      if (ms) {
        self_seen = true;
        self_kept = total + __popc(m & (ms - 1u)) < cap;
      }
      total += __popc(m);
      if (m) last = c0 + 31 - __clz(m);
    }
  }
  acc = min(total, cap);
  cnt = acc - (self_kept ? 1 : 0);
  cand = W;
  trunc = total > cap || (total == cap && last < W - 1);
}

// A lane's accepted entries wait in shared memory (kListWait rows of 32
// lanes) until some lane of the warp has no room for its next tile, and then
// go out in chunks of four: an entry costs a leading-zero count, a mask, a
// load and a store, 9 instructions where collecting four in registers and
// testing for a full chunk took about 25 and was half of the pass (a warp
// waits in every tile for the lane with the most hits).
constexpr int kListWait = 36;   // a tile's 32 and the up to 3 of an unfinished chunk

// What a warp stages: the next candidates to be screened, a ring of two
// tiles (negated x, y, z in the frame of the group's lowest cell, the list
// entry, the z cell less that cell's predecessor), where the lanes' own
// particles went, and each z cell's candidates of a tile.
struct ListStage {
  float nx[64], ny[64], nz[64];
  int entry[64];
  unsigned kmask[32];
  int self_at[32];
  unsigned char krel[64];
};

// The neighbour lists.  The lanes of a warp whose particles share a column of
// cells, up to SPAN z cells apart, form a group.  The runs of the group's
// common window are read as one sequence, 32 candidates at a time; the lane
// that reads a candidate drops it if it is farther than 2h from the box around
// the group's particles (a fifth of a dense 3D window: its edges and corners),
// and what is left fills tiles of 32 across the runs, which every lane screens
// (screen_tile).  A dense 3D group takes 16 tiles where a tile for each part of
// each run took 27.
//
// Bound by latency: a warp waits for its own shared memory, shuffles and
// results (6.7 of an instruction's 7.7 warp-cycles at 256,000 particles, with 4.3
// warps a scheduler; issue slots 57% busy, no pipe above 44%), in small
// simulations for its chain of tiles.  Blocks of two warps: small simulations spread over the SMs, and a
// block does not wait for its slowest of eight warps.  Registers decide the
// rest: 96 in 3D and 80 in 2D (9 and 12 blocks an SM asked for) keep the loop
// out of local memory and beat fewer and more (box of 10^6, 8, 9, 12 and 16
// blocks: 630, 568, 598 and 675 us; 2D, 1.02 10^6 particles, 9, 12 and 16:
// 137, 122 and 131).  Against one tile for each run part and eight warps a
// block, on one B200: 735 -> 568 us for that box, 483 -> 379 at 864,000
// particles of the dam break, 68 -> 53 at 62,500, 157 -> 96 at 94,221 (columns
// of about a warp's particles, where a warp spans a whole column), 133 -> 122
// in 2D.
constexpr int kListBlock = 64;

template <int DIM>
__global__ void __launch_bounds__(kListBlock, DIM == 3 ? 9 : 12) k_neighbour_lists(DevBatch b) {
  chain_wait();
  constexpr int T = kListBlock, PARTS = kBlock / T;   // a tile's parts
  constexpr int NR = (DIM == 3) ? 9 : 3, RY = (DIM == 3) ? 3 : 1, SPAN = (DIM == 3) ? 9 : kMostSpan;
  static_assert((SPAN + 1) * RY <= 32, "one lane for each z cell and y column");
  __shared__ SimDev s;
  __shared__ __align__(16) ListStage stage[T / 32];
  __shared__ int wait[T / 32][kListWait][32];
  __shared__ __align__(16) ListRun run_table[T / 32][NR];
  int cur = -1;
  const Particles& P = b.P;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned FULL = 0xffffffffu, below = (1u << lane) - 1u;
  ListStage& g = stage[warp];
  ListRun* const runs = run_table[warp];
  int* const mine_wait = &wait[warp][0][lane];
  const int alone = b.ntiles < 2 * b.sms ? 20 : 6;   // quarters: the weight of a particle taken singly
  for (int t = blockIdx.x; t < b.ntiles * PARTS; t += gridDim.x) {
    const Tile tl = b.tiles[t / PARTS];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    const int at = (t % PARTS) * T + threadIdx.x;
    const int p = tl.start + at;
    const bool active = at < tl.count && p < s.p_off + dyn->nag && !dyn->frozen;
    float4 xf = make_float4(0.f, 0.f, 0.f, 0.f);
    int ci = 0, cj = 0, ck = 0;
    bool on = false;
    if (active) {
      const double4 xd = P.X[p];
      xf = P.XF[p];
      on = particle_cell(s, xd.x, xd.y, xd.z, ci, cj, ck);
      if (!on) set_status(dyn, SPH_ERR_INVALID_ARGUMENT);   // state not re-sorted after a move
    }
    const int colkey = on ? (cj * s.ncd[0] + ci) : -1;
    unsigned remaining = __ballot_sync(FULL, on);
    int done = 0, n = 0, nacc = 0, cand = 0;         // entries written, waiting; accepted, candidates
    bool trunc = false;
    const int cap = s.nmaxpartj;
    int4* out = reinterpret_cast<int4*>(b.nlist) + list_base4(p, b.list_cap4);
    const float mid = 0.5f * (s.rr_lo + s.rr_hi), delta = 0.5f * (s.rr_hi - s.rr_lo) * 1.01f, dz = s.dcdf[2];
    // the waiting chunks of all lanes; what is left moves to the front
    auto flush = [&]() {
      const int chunks = n >> 2;
      const int most = (int)__reduce_max_sync(FULL, (unsigned)chunks);
      int4* o = out + (size_t)(done >> 2) * 32;
      for (int k = 0; k < most; ++k) {
        if (k < chunks) {
          const int* e = mine_wait + 128 * k;
          o[(size_t)k * 32] = make_int4(e[0], e[32], e[64], e[96]);
        }
      }
      const int* e = mine_wait + 128 * chunks;
      const int left = n & 3;
      if (left > 0) mine_wait[0] = e[0];
      if (left > 1) mine_wait[32] = e[32];
      if (left > 2) mine_wait[64] = e[64];
      done += 4 * chunks;
      n = left;
    };
    while (remaining) {
      const int leader = __ffs(remaining) - 1;
      const int key = __shfl_sync(FULL, colkey, leader);
      bool mine = ((remaining >> lane) & 1u) && colkey == key;
      const int kmin = __reduce_min_sync(FULL, mine ? ck : 0x7fffffff);
      mine = mine && ck - kmin <= SPAN;
      const int kmax = __reduce_max_sync(FULL, mine ? ck : -0x7fffffff);
      const unsigned group = __ballot_sync(FULL, mine);
      remaining &= ~group;
      const int gci = __shfl_sync(FULL, ci, leader);
      const int gcj = __shfl_sync(FULL, cj, leader);
      // the runs of the common window, and each z cell's candidates
      const int klo = kmin > 1 ? kmin - 1 : 1, khi = kmax < s.ncd[2] ? kmax + 1 : s.ncd[2];
      int ub = 0, ue = 0;
      if (lane < NR) {
        const int jr = (DIM == 3) ? gcj - 1 + lane / 3 : gcj, ir = gci - 1 + ((DIM == 3) ? lane % 3 : lane);
        if (ir >= 1 && ir <= s.ncd[0] && jr >= 1 && jr <= s.ncd[1]) {
          const int base = s.cell_off + ((jr - 1) * s.ncd[0] + (ir - 1)) * s.ncd[2];
          ub = __ldg(P.cell_start + base + klo - 1);
          ue = __ldg(P.cell_start + base + khi);
        }
      }
      int part = 0;
      {
        const int k = kmin + lane / RY, jr = (DIM == 3) ? gcj - 1 + lane % RY : gcj;
        if (k <= kmax && jr >= 1 && jr <= s.ncd[1]) {
          const int ml = k > 1 ? k - 1 : 1, mh = k < s.ncd[2] ? k + 1 : s.ncd[2];
#pragma unroll
          for (int x = -1; x <= 1; ++x) {
            if (gci + x < 1 || gci + x > s.ncd[0]) continue;
            const int base = s.cell_off + ((jr - 1) * s.ncd[0] + (gci + x - 1)) * s.ncd[2];
            part += __ldg(P.cell_start + base + mh) - __ldg(P.cell_start + base + ml - 1);
          }
        }
      }
      int inc = ue - ub;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const int v = __shfl_up_sync(FULL, inc, o, 16);
        if ((lane & 15) >= o) inc += v;
      }
      const int W = __shfl_sync(FULL, inc, NR - 1);
      {
        const int kr = mine ? (ck - kmin) * RY : 0;
        int c = __shfl_sync(FULL, part, kr);
        if (DIM == 3) c += __shfl_sync(FULL, part, kr + 1) + __shfl_sync(FULL, part, kr + 2);
        if (mine) cand = c;
      }
      // few lanes, or a common window many times their own: a particle at a
      // time (list_by_ballots).  Both sides are instruction counts: 160 and
      // one a candidate for a particle, 256 and eight a candidate for the
      // group's window, a particle's weighted 1.5 (127,008 particles: 133 us
      // with 1, 128 with 1.5; 176,435: 126 and 109) and, where an SM has few
      // warps and each waits for its own loads, 5 (13,500 particles: 60 us
      // with groups of up to 7 taken singly, 47 with up to 2).
      if (__popc(group) * (160 + __shfl_sync(FULL, cand, leader)) * alone < 4 * (256 + 8 * W)) {
        for (unsigned left = group; left; left &= left - 1) {
          const int o = __ffs(left) - 1;
          const float4 xo = make_float4(__shfl_sync(FULL, xf.x, o), __shfl_sync(FULL, xf.y, o),
                                        __shfl_sync(FULL, xf.z, o), 0.f);
          int cn, ac, ca;
          bool tr;
          list_by_ballots<DIM>(s, b, p - lane + o, xo, gci, gcj, __shfl_sync(FULL, ck, o), runs, cn, ac, ca, tr);
          if (lane == o) {
            done = cn;
            nacc = ac;
            cand = ca;
            trunc = tr;
          }
        }
        continue;
      }
      __syncwarp();
      if (lane < NR)
        runs[lane] = ListRun{inc, ub - (inc - (ue - ub)), (float)(((DIM == 3) ? lane % 3 : lane) - 1) * s.dcdf[0],
                             (DIM == 3) ? (float)(lane / 3 - 1) * s.dcdf[1] : 0.f};
      g.self_at[lane] = -1;
      // the box of the group's particles, offsets from its lowest cell's
      // origin (not below 0: float bits order as integers), and the distance
      // beyond which no lane's FP32 value can be within the band
      const float zi = (float)(ck - kmin) * dz + xf.z;
      const int far_lo = 0x7f000000;
      const float bx0 = __int_as_float(__reduce_min_sync(FULL, mine ? __float_as_int(fmaxf(xf.x, 0.f)) : far_lo));
      const float bx1 = __int_as_float(__reduce_max_sync(FULL, mine ? __float_as_int(fmaxf(xf.x, 0.f)) : 0));
      const float bz0 = __int_as_float(__reduce_min_sync(FULL, mine ? __float_as_int(fmaxf(zi, 0.f)) : far_lo));
      const float bz1 = __int_as_float(__reduce_max_sync(FULL, mine ? __float_as_int(fmaxf(zi, 0.f)) : 0));
      float by0 = 0.f, by1 = 0.f;
      if (DIM == 3) {
        by0 = __int_as_float(__reduce_min_sync(FULL, mine ? __float_as_int(fmaxf(xf.y, 0.f)) : far_lo));
        by1 = __int_as_float(__reduce_max_sync(FULL, mine ? __float_as_int(fmaxf(xf.y, 0.f)) : 0));
      }
      const float far2 = s.rr_hi * 1.001f;
      int at_cap = 0;                                // the entry at which a lane reached NMAXPARTJ
      __syncwarp();
      // one tile of nt staged candidates, the first of them number c0
      auto tile = [&](int c0, int nt) {
        const int h = c0 & 32;
        float near = 3.0e38f;
        unsigned hitm = screen_tile<DIM>(g.nx + h, g.ny + h, g.nz + h, nt, xf.x, xf.y, zi, mid, near);
        if (!mine) hitm = 0u;
        // only the lane's own window counts: the group's common window
        // reaches beyond some lanes', and where the cells are narrower than
        // 2h (CreaGrid rounds the cell count to nearest) a candidate there
        // can lie within 2h without being the reference's neighbour; with
        // cells at least 2h wide such a candidate is never a hit below the
        // band, and band hits are tested below
        if (s.narrow_z) {
          g.kmask[lane] = 0u;
          __syncwarp();
          const int kr = lane < nt ? g.krel[h + lane] & 31 : 31;
          g.kmask[kr] = __brev(__match_any_sync(FULL, kr));
          __syncwarp();
          const unsigned* w = g.kmask + (mine ? ck - kmin : 0);
          hitm &= w[0] | w[1] | w[2];
        }
        if (mine && near <= delta) {
          // rare: candidates in the band -- outside the lane's window (the
          // reference never visits those) or failing the FP64 test they
          // are dropped; hitm then holds exactly the accepted ones
          for (int u = 0; u < nt; ++u) {
            const float d0 = xf.x + g.nx[h + u], d1 = (DIM == 3) ? xf.y + g.ny[h + u] : 0.f, d2 = zi + g.nz[h + u];
            float rr = __fmul_rn(d0, d0);
            if (DIM == 3) rr = __fmaf_rn(d1, d1, rr);
            rr = __fmaf_rn(d2, d2, rr);
            if (!(fabsf(rr - mid) <= delta)) continue;
            const int slot = g.entry[h + u] & kSlotMask;
            bool keep = fabsf(P.XF[slot].w - (float)ck) <= 1.0f;
            if (keep) {
              const double4 xq = P.X[slot], xi = P.X[p];
              const double r0 = xi.x - xq.x, r1 = xi.y - xq.y, r2 = xi.z - xq.z;
              keep = !(r0 * r0 + r1 * r1 + r2 * r2 > s.square_doubleh);
            }
            const unsigned bit = 0x80000000u >> u;
            hitm = keep ? (hitm | bit) : (hitm & ~bit);
          }
        }
        if (nacc >= cap) hitm = 0u;                  // NMAXPARTJ reached: every later candidate is refused
        const int more = __popc(hitm);
        if (nacc + more >= cap && more > 0) {
          // reaching NMAXPARTJ in this tile (rare): the accepted ones in
          // visiting order up to the cap, candidate u the last of them
          int u = 0, left = cap - nacc;
          unsigned m = hitm;
#pragma unroll
          for (int w = 16; w > 0; w >>= 1) {
            const int c = __popc(m >> (32 - w));
            if (c < left) {
              left -= c;
              m <<= w;
              u += w;
            }
          }
          hitm &= ~(0x7fffffffu >> u);
          nacc = cap;
          at_cap = g.entry[h + u];
        } else {
          nacc += more;
        }
        // the lane itself: counted, not stored
        const unsigned self = (unsigned)(g.self_at[lane] - c0);
        if (self < 32u) hitm &= ~(0x80000000u >> self);
        const int add = __popc(hitm);
        if (__any_sync(FULL, n + add > kListWait)) flush();
        int* dst = mine_wait + 32 * n;
        n += add;
        const int* ent = g.entry + h;
        while (hitm) {
          const int u = __clz(hitm);
          hitm &= 0x7fffffffu >> u;
          *dst = ent[u];
          dst += 32;
        }
      };
      int staged = 0, screened = 0, r = 0, e = -1;
      float4 f;
      float dx = 0.f, dy = 0.f;
      auto fetch = [&](int c) {                      // candidate c of the runs
        e = -1;
        if (c < W) {
          while (c >= runs[r].end) ++r;
          const ListRun q = runs[r];
          e = (q.base + c) | (r << kSlotBits);
          dx = q.dx;
          dy = q.dy;
          f = __ldg(P.XF + (q.base + c));
        }
      };
      fetch(lane);
      for (int c = lane; c - lane < W; c += 32) {
        const int e0 = e;
        bool keep = false;
        float x = 0.f, y = 0.f, z = 0.f;
        int kr = 0;
        if (e0 != -1) {
          x = f.x + dx;
          y = f.y + dy;
          z = (f.w - (float)kmin) * dz + f.z;
          kr = (int)f.w - kmin + 1;
          const float gx = fmaxf(fmaxf(bx0 - x, x - bx1), 0.f), gz = fmaxf(fmaxf(bz0 - z, z - bz1), 0.f);
          float d = __fmaf_rn(gx, gx, gz * gz);
          if (DIM == 3) {
            const float gy = fmaxf(fmaxf(by0 - y, y - by1), 0.f);
            d = __fmaf_rn(gy, gy, d);
          }
          keep = d <= far2;
        }
        fetch(c + 32);
        const unsigned m = __ballot_sync(FULL, keep);
        const int pos = staged + __popc(m & below), w = pos & 63;
        if (keep) {
          g.nx[w] = -x;
          g.ny[w] = -y;
          g.nz[w] = -z;
          g.entry[w] = e0;
          if (s.narrow_z) g.krel[w] = (unsigned char)kr;
          const unsigned o = (unsigned)((e0 & kSlotMask) - (p - lane));
          if (o < 32u && (int)((unsigned)e0 >> kSlotBits) == NR / 2) g.self_at[o] = pos;
        }
        staged += __popc(m);
        __syncwarp();
        if (staged - screened >= 32) {
          tile(screened, 32);
          screened += 32;
          __syncwarp();
        }
      }
      if (staged > screened) {
        const int nt = staged - screened, w = (screened & 32) + lane;
        if (lane >= nt) {
          g.nx[w] = -3.0e18f;
          g.ny[w] = -3.0e18f;
          g.nz[w] = -3.0e18f;
        }
        __syncwarp();
        tile(screened, nt);
      }
      if (mine && nacc >= cap) {
        // whether candidates of the window follow the one that reached the
        // cap: here for all lanes at a time, not for a tile's few lanes each
        // (200,000 particles cut to 43 of 74 neighbours: 204 us so, 191 here)
        int seen = 0;
        if (cap > 0) {
          const int last = (int)((unsigned)at_cap >> kSlotBits);
          const int ml = ck > 1 ? ck - 1 : 1, mh = ck < s.ncd[2] ? ck + 1 : s.ncd[2];
          for (int q = 0; q <= last; ++q) {
            const int jr = (DIM == 3) ? gcj - 1 + q / 3 : gcj, ir = gci - 1 + ((DIM == 3) ? q % 3 : q);
            if (ir < 1 || ir > s.ncd[0] || jr < 1 || jr > s.ncd[1]) continue;
            const int base = s.cell_off + ((jr - 1) * s.ncd[0] + (ir - 1)) * s.ncd[2];
            seen += (q == last ? (at_cap & kSlotMask) + 1 : P.cell_start[base + mh]) - P.cell_start[base + ml - 1];
          }
        }
        trunc = seen < cand;
      }
      __syncwarp();
    }
    flush();
    if (n > 0) {
      // the last, partial chunk
      int4 w = make_int4(mine_wait[0], 0, 0, 0);
      if (n > 1) w.y = mine_wait[32];
      if (n > 2) w.z = mine_wait[64];
      out[(size_t)(done >> 2) * 32] = w;
    }
    if (active) b.ncount[p] = done + n;
    // one per warp: every cut particle's own met the others at one address
    // (the same 200,000: 187 us so, 120 here)
    if (__any_sync(FULL, trunc) && lane == 0) atomicOr(&dyn->warnings, SPH_WARN_NEIGHBOURS_TRUNCATED);
    block_count2(b.counters, cand, nacc);
    const int m = warp_max(nacc);
    if (lane == 0 && m > 0) atomicMax(&dyn->max_neigh, m);
  }
}

// ==========================================================================
// Momentum, FP64 form: RHS_momentum_equation + inter_EqMoto + viscomon +
// viscomorris + AddBoundaryContributions_to_ME3D/2D +
// AddElasticBoundaryReaction_3D/2D, optionally fused with Leapfrog_momentum,
// velocity_smoothing_2 (TetaV = 0), Leapfrog_trajectories and the CFL part of
// time_step_duration.  The list is drained in warp lockstep.
// ==========================================================================
// CalcVarLength.f90:285-324 (3D, C1_BE): the fluid part of the
// renormalisation matrices, summed over the particle's list in its order.
// A pair adds (x_j - x_i)_c grad_W_k m_j / rho_j to B(k,c), grad_W that of
// the anti-cluster kernel for B_ren_gradp and of the beta-spline for
// B_ren_divu (grad_W_sub.f90:52-91, 3D); a pair with r >= 2h adds nothing
// (CalcVarLength.f90:254), nor does a zero gradient (r < 1e-6 h, the
// particle itself): the sums start at +0, so skipping a +-0 addend leaves
// them as they are.  The frontier terms are added by the momentum (first
// step) and continuity passes, which also invert.  One sqrt and the
// division r / h are shared by the range test and both gradients; the
// constant factors come from the host (SimDev::c1_w*).  The pair's twelve
// divisions by |r| and rho_j go through one correctly rounded reciprocal
// of each (the IEEE quotients; the sums start at +0, so the sign of a zero
// term is of no account).
// The 2D SA-SPH frontier terms of the renormalisation matrices, -RN IntWdV
// per close side (AddBoundaryContribution_to_CE2D.f90:81-94 for both
// matrices in every continuity pass; AddBoundaryContributions_to_ME2D.f90:
// 290-300 for B_ren_gradp on the first step, GRADP_ONLY), then their
// inversion (SASPH_continuity.f90:112-119, ME2D.f90:377-383).  In 2D the
// matrices have a zero y row and column, so their determinant is zero and
// the inversion always gives the -I of B_ren_gradp_inversion.f90:67-72
// (a positive invb_det_thresh is required); renormalising with -I leaves
// every vector as it is, so the rates are the plain form's and only the
// matrices themselves are formed here.
template <bool GRADP_ONLY>
__global__ void k_c1_frontier_2d(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  const int total = P.total_slots;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    const SimDyn* dyn = b.dyn + tl.sim;
    if (!s.c1_be || dyn->frozen || (GRADP_ONLY && dyn->step != 0)) continue;
    const int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + dyn->nag) continue;
    const bool divu = !GRADP_ONLY && s.c1_divu;
    double Bg[9], Bd[9];
    load_b(P.BG, total, p, Bg);
    if (divu) load_b(P.BD, total, p, Bd);
    const int nb = P.bdt_count[p];
    const int start = nb > 0 ? P.bdt_start[p] : 0;
    for (int u = 0; u < nb; ++u) {
      const BdtEntry& e = P.bdt[start + u];
      const SideDev& S = b.sides[s.side_off + e.clobonum - 1];
      const double IntWdV = e.bi[2];
      const int ax[2] = {0, 2};
      for (int a = 0; a < 2; ++a)
        for (int c = 0; c < 2; ++c) {
          const double aux = -S.RN[a][c] * IntWdV;
          Bg[3 * ax[a] + ax[c]] = Bg[3 * ax[a] + ax[c]] + aux;
          if (divu) Bd[3 * ax[a] + ax[c]] = Bd[3 * ax[a] + ax[c]] + aux;
        }
    }
    if (divu) {
      b_inversion(Bd, s.invb_det_thresh);
      store_b(P.BD, total, p, Bd);
    }
    b_inversion(Bg, s.invb_det_thresh);
    store_b(P.BG, total, p, Bg);
  }
}

// 2D (DIM = 2): grad_W_sub.f90:79-88 scales both gradients by h 10/7
// (beta-spline) and h 4/3 (anti-cluster); y is zero throughout.
template <int DIM>
__global__ void __launch_bounds__(kBlock, 2) k_renormalisation(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  const int total = P.total_slots;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    if (!s.c1_be) continue;
    const bool divu = s.c1_divu != 0;
    int p = tl.start + threadIdx.x;
    bool active = threadIdx.x < tl.count && p < s.p_off + b.dyn[tl.sim].nag;
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    int cnt = 0;
    if (active) {
      xi = P.X[p];
      cnt = b.ncount[p];
    }
    double Bg[9], Bd[9];
    for (int k = 0; k < 9; ++k) Bg[k] = Bd[k] = 0.0;
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    for (int k = 0; k < nmax; ++k) {
      int e = lr.get(k);
      if (k >= cnt) continue;
      int q = e & kSlotMask;
      const double4 xj = load_record(P.X + q);
      double r[3] = {xj.x - xi.x, xj.y - xi.y, xj.z - xi.z};
      double abs_r = sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]);
      double qh = div_rn_unsigned0(abs_r, s.h, s.rcp_h);
      if (at_least_two(qh) || abs_r < s.h * 1.0e-6) continue;
      const double mj = xj.w, rhoj = P.RP[q].x;
      const double w = 2.0 - qh;
      double go[3];
      // anti-cluster kernel (q <= 2 here)
      const double rcp_r = __drcp_rn(abs_r), rcp_rhoj = __drcp_rn(rhoj);
      double t = div_rn_unsigned0(-(3.0 * (w * w) * s.c1_w2), s.h, s.rcp_h);
      for (int c = 0; c < 3; ++c) {
        double gw = div_rn_unsigned0(t * r[c], abs_r, rcp_r);
        if (DIM == 2) gw = gw * s.h * 4.0 / 3.0;
        go[c] = div_rn_unsigned0(gw * mj, rhoj, rcp_rhoj);
      }
      for (int c = 0; c < 3; ++c)
        for (int kk = 0; kk < 3; ++kk) Bg[3 * kk + c] = Bg[3 * kk + c] + r[c] * go[kk];
      if (divu) {
        // beta-spline (q < 2 here)
        t = div_rn_unsigned0(qh <= 1.0 ? s.c1_w1a * (9.0 / 4.0 * (qh * qh) - 3.0 * qh) : -(s.c1_w1b * (w * w)), s.h, s.rcp_h);
        for (int c = 0; c < 3; ++c) {
          double gw = div_rn_unsigned0(t * r[c], abs_r, rcp_r);
          if (DIM == 2) gw = gw * s.h * 10.0 / 7.0;
          go[c] = div_rn_unsigned0(gw * mj, rhoj, rcp_rhoj);
        }
        for (int c = 0; c < 3; ++c)
          for (int kk = 0; kk < 3; ++kk) Bd[3 * kk + c] = Bd[3 * kk + c] + r[c] * go[kk];
      }
    }
    if (active) {
      store_b(P.BG, total, p, Bg);
      if (divu) store_b(P.BD, total, p, Bd);
    }
  }
}

// A particle of a finished simulation of a batch: its record as it is, for
// the step's sort.
__device__ __forceinline__ void carry_record(const Particles& P, int p) {
  const double4 v4 = P.V[p];
  const double2 rp = P.RP[p];
  P.X2[p] = P.X[p];
  P.V2[p] = make_double4(v4.x, v4.y, v4.z, rp.x);
  P.P2[p] = rp.y;
  P.I2[p] = P.I[p];
  P.L2[p] = P.L[p];
}

// The particle's values that its pairs share.
struct PairSelf {
  double4 x;
  double v[3];
  double rho, p, rcp_rho, mon;   // mon: alfa_mon (2 c) h
  bool morris;
  double nu;
  __device__ __forceinline__ void load(const SimDev& s, const double4& xi, const double4& vi, double rhoi, double pi) {
    x = xi;
    v[0] = vi.x;
    v[1] = vi.y;
    v[2] = vi.z;
    rho = rhoi;
    p = pi;
    rcp_rho = __drcp_rn(rhoi);
    mon = s.alfa_mon * (s.celerita + s.celerita) * s.h;
    nu = s.kin_visc;
    morris = nu > 1.0e-12;
  }
};

// One pair's terms of the momentum equation, component d handed to
// add(kind, d, term) as each is formed: kind 0 the pressure gradient, 1 ALE1
// (to be taken from its sum), 2 Monaghan's and 3 Morris's viscosity.
template <int DIM, class ADD>
__device__ __forceinline__ void pair_terms(const SimDev& s, const PairSelf& i, const double4& xj, const double4& vj,
                                           const double2& rpj, ADD&& add) {
  double r0 = i.x.x - xj.x, r1 = i.x.y - xj.y, r2 = i.x.z - xj.z;
  double rr = r0 * r0 + r1 * r1 + r2 * r2;
  double PK1, PK2, PK3;
  kernel_values(s, rr, PK1, PK2, PK3);
  double rhoj = rpj.x, pj = rpj.y, amassj = xj.w;
  double dv0 = vj.x - i.v[0], dv1 = vj.y - i.v[1], dv2 = vj.z - i.v[2];
  // pressure gradient and ALE1 terms, inter_EqMoto.f90:195-221
  // the two divisions by rho_i rho_j and the one by rho_i share correctly
  // rounded reciprocals (the IEEE quotients; the sums start at +0, so the
  // sign of a zero term is of no account)
  const double rr_ij = i.rho * rhoj, rcp_rr = __drcp_rn(rr_ij);
  double alpha = div_rn_unsigned0(pj - i.p, rr_ij, rcp_rr);
  add(0, 0, -(amassj * alpha * r0 * PK3));
  if (DIM == 3) add(0, 1, -(amassj * alpha * r1 * PK3));
  add(0, 2, -(amassj * alpha * r2 * PK3));
  double alpha2 = div_rn_unsigned0(i.p * (div_rn_unsigned0(rhoj, i.rho, i.rcp_rho) + 1.0) + pj * (i.rho / rhoj - 1.0),
                                   rr_ij, rcp_rr);
  add(1, 0, amassj * alpha2 * r0 * PK3);
  if (DIM == 3) add(1, 1, amassj * alpha2 * r1 * PK3);
  add(1, 2, amassj * alpha2 * r2 * PK3);
  // viscomon.f90:54-73
  double vrij = (DIM == 3) ? -(dv0 * r0) - dv1 * r1 - dv2 * r2 : -(dv0 * r0) - dv2 * r2;
  double TermMon = i.mon / (i.rho + rhoj);
  double mtv = amassj * TermMon * vrij;
  add(2, 0, mtv * r0 * PK2 + 0.0);
  if (DIM == 3) add(2, 1, mtv * r1 * PK2 + 0.0);
  add(2, 2, mtv * r2 * PK2 + 0.0);
  // viscomorris.f90:60-71
  if (i.morris) {
    double rt = i.nu * i.rho + i.nu * rhoj + 1.0e-3;
    double anuitilde = 4.0 * (i.nu * i.nu);
    double factivis = amassj * anuitilde / rt;
    add(3, 0, factivis * (-(dv0 * PK2 * rr)));
    if (DIM == 3) add(3, 1, factivis * (-(dv1 * PK2 * rr)));
    add(3, 2, factivis * (-(dv2 * PK2 * rr)));
  }
}

// The closing of an FP64 momentum pass for particle p from its sums: the
// laminar flag, gravity, the elastic reaction and, in the fused step, the
// leapfrog update and the particle's CFL time.
template <int DIM, bool FUSED>
__device__ __forceinline__ void momentum_close(const SimDev& s, const DevBatch& b, SimDyn* dyn, int p,
                                               const double4& xi, const double* vi, double rhoi, double pi,
                                               const double* tpres, const double* td, const double* tv,
                                               const double* rs, double& dtc) {
  const Particles& P = b.P;
  const double GI = (double)9.80665f;   // Static_allocation_module.f90:72, a default-REAL literal
  const double* geff = dyn->geff;
  const int nb = P.bdt_count[p];
  const int bstart = nb > 0 ? P.bdt_start[p] : 0;
  // laminar_flag, inter_EqMoto.f90:269-283
  int lam_new = 0;
  if (s.kin_visc > 0.0) {
    double absv_pres = sqrt(tpres[0] * tpres[0] + tpres[1] * tpres[1] + tpres[2] * tpres[2]) + GI;
    double absv_morris = sqrt(rs[0] * rs[0] + rs[1] * rs[1] + rs[2] * rs[2]);
    double weight = 0.0;
    if (absv_pres != 0.0) weight = absv_morris / absv_pres * 100.0;
    lam_new = (weight > 5.0 || absv_pres == 0.0) ? 1 : 0;
  }
  double acc[3];
  acc[0] = tpres[0] + td[0] + tv[0] + geff[0];
  acc[1] = tpres[1] + td[1] + tv[1] + geff[1];
  acc[2] = tpres[2] + td[2] + tv[2] + geff[2];
  if (nb > 0) {
    double R[3];
    const double xa[3] = {xi.x, xi.y, xi.z};
    elastic_reaction<DIM>(s, b, nb, bstart, xa, vi, R);
    for (int d = 0; d < 3; ++d) acc[d] = acc[d] + R[d];
  }
  if (FUSED) {
    double dtvel = dyn->dtvel, dt = dyn->dt;
    double vn[3], xn[3];
    for (int d = 0; d < 3; ++d) vn[d] = vi[d] + dtvel * acc[d];
    xn[0] = xi.x + dt * vn[0];
    xn[1] = xi.y + dt * vn[1];
    xn[2] = xi.z + dt * vn[2];
    P.X2[p] = make_double4(xn[0], xn[1], xn[2], xi.w);
    P.V2[p] = make_double4(vn[0], vn[1], vn[2], rhoi);
    P.P2[p] = pi;
    P.I2[p] = P.I[p];
    P.L2[p] = (uint8_t)lam_new;
    double U = sqrt(vn[0] * vn[0] + vn[1] * vn[1] + vn[2] * vn[2]);
    // with velocity smoothing the CFL minimum is taken on the smoothed
    // velocities (k_velocity_smoothing_apply), which also moves X2
    if (!(s.teta_v > 1.0e-9)) dtc = s.cfl * 2.0 * s.h / (s.celerita + U);
  } else {
    P.ACC[p] = make_double4(acc[0], acc[1], acc[2], 0.0);
    P.L[p] = (uint8_t)lam_new;
  }
}

// C1: with input_any_t%C1_BE the pressure terms are renormalised with
// B_ren_gradp (3D only).
// BATCH (not with C1): two list entries' records are requested before the
// first one's arithmetic, so the second pair's gathers wait behind the
// first pair's FP64 divisions instead of after them; the terms are formed
// and summed in the same order, so the results are the same bits.
template <int DIM, bool FUSED, bool C1 = false, bool BATCH = false>
__global__ void __launch_bounds__(kBlock, 2) k_momentum(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  __shared__ double stpres[3][kBlock];   // the wall pressure term, kept out of the pair loop's registers
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    const double* geff = dyn->geff;
    int p = tl.start + threadIdx.x;
    bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag;
    if (FUSED && active && dyn->frozen) {
      carry_record(P, p);
      active = false;
    }
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    double vi[3] = {0.0, 0.0, 0.0};
    double rhoi = 1.0, pi = 0.0;
    int cnt = 0;
    double tdiss[3] = {0, 0, 0}, tvisc[3] = {0, 0, 0};
    if (active) {
      xi = P.X[p];
      double4 v4 = P.V[p];
      double2 rp = P.RP[p];
      vi[0] = v4.x;
      vi[1] = v4.y;
      vi[2] = v4.z;
      rhoi = rp.x;
      pi = rp.y;
      cnt = b.ncount[p];
      const int nb = P.bdt_count[p];
      double tpres[3] = {0, 0, 0};
      // C1: on the first step the frontiers complete B_ren_gradp and it is
      // inverted, for every particle (RHS_momentum_equation.f90:130-150)
      const bool c1 = C1 && s.c1_be;
      const bool first = c1 && dyn->step == 0;
      if (c1) {
        double B[9];
        load_b(P.BG, P.total_slots, p, B);
        if (nb > 0)
          me_boundary3d<true>(s, b, nb, P.bdt_start[p], vi, rhoi, pi, P.L[p], geff, tpres, tdiss, tvisc, B, first);
        else if (first)
          b_inversion(B, s.invb_det_thresh);
        if (first) store_b(P.BG, P.total_slots, p, B);
      } else if (nb > 0) {
        const int lam = P.L[p];
        const int bstart = P.bdt_start[p];
        if (DIM == 3) me_boundary3d(s, b, nb, bstart, vi, rhoi, pi, lam, geff, tpres, tdiss, tvisc);
        else me_boundary2d(s, b, nb, bstart, vi, rhoi, pi, lam, geff, tpres, tdiss, tvisc);
      }
      for (int d = 0; d < 3; ++d) stpres[d][threadIdx.x] = tpres[d];
    }
    double tp0 = 0, tp1 = 0, tp2 = 0, al0 = 0, al1 = 0, al2 = 0;
    double td0 = tdiss[0], td1 = tdiss[1], td2 = tdiss[2];
    double tv0 = tvisc[0], tv1 = tvisc[1], tv2 = tvisc[2];
    double rs0 = 0, rs1 = 0, rs2 = 0;
    PairSelf self;
    self.load(s, xi, make_double4(vi[0], vi[1], vi[2], 0.0), rhoi, pi);
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    auto pair = [&](const double4& xj, const double4& vj, const double2& rpj) {
      pair_terms<DIM>(s, self, xj, vj, rpj, [&](int kind, int d, double a) {
        if (kind == 0) {
          if (d == 0) tp0 = tp0 + a;
          else if (d == 1) tp1 = tp1 + a;
          else tp2 = tp2 + a;
        } else if (kind == 1) {
          if (d == 0) al0 = al0 - a;
          else if (d == 1) al1 = al1 - a;
          else al2 = al2 - a;
        } else if (kind == 2) {
          if (d == 0) td0 = td0 + a;
          else if (d == 1) td1 = td1 + a;
          else td2 = td2 + a;
        } else {
          if (d == 0) tv0 = tv0 + a, rs0 = rs0 + a;
          else if (d == 1) tv1 = tv1 + a, rs1 = rs1 + a;
          else tv2 = tv2 + a, rs2 = rs2 + a;
        }
      });
    };
    if (BATCH) {
      for (int k = 0; k < nmax; k += 2) {
        const int e0 = lr.get(k);
        const int e1 = k + 1 < nmax ? lr.get(k + 1) : 0;
        const bool u0 = k < cnt, u1 = k + 1 < cnt;
        double4 x0 = make_double4(0.0, 0.0, 0.0, 0.0), v0 = x0, x1 = x0, v1 = x0;
        double2 p0 = make_double2(0.0, 0.0), p1 = p0;
        if (u0) {
          const int q = e0 & kSlotMask;
          x0 = load_record(P.X + q); v0 = load_record(P.V + q); p0 = __ldg(P.RP + q);
        }
        if (u1) {
          const int q = e1 & kSlotMask;
          x1 = load_record(P.X + q); v1 = load_record(P.V + q); p1 = __ldg(P.RP + q);
        }
        if (u0) pair(x0, v0, p0);
        if (u1) pair(x1, v1, p1);
      }
    } else {
      for (int k = 0; k < nmax; ++k) {
        int e = lr.get(k);
        if (k >= cnt) continue;
        int q = e & kSlotMask;
        pair(load_record(P.X + q), load_record(P.V + q), __ldg(P.RP + q));
      }
    }
    double dtc = 1.0e300;
    if (active) {
      if (C1 && s.c1_be) {
        // inter_EqMoto.f90:255-260
        double B[9], tp[3] = {tp0, tp1, tp2};
        load_b(P.BG, P.total_slots, p, B);
        b_renormalise(B, tp);
        tp0 = tp[0];
        tp1 = tp[1];
        tp2 = tp[2];
      }
      double tpres[3];
      tpres[0] = stpres[0][threadIdx.x] + tp0 + al0;
      tpres[1] = stpres[1][threadIdx.x] + tp1 + al1;
      tpres[2] = stpres[2][threadIdx.x] + tp2 + al2;
      const double td[3] = {td0, td1, td2}, tv[3] = {tv0, tv1, tv2}, rs[3] = {rs0, rs1, rs2};
      momentum_close<DIM, FUSED>(s, b, dyn, p, xi, vi, rhoi, pi, tpres, td, tv, rs, dtc);
    }
    if (FUSED) {
      double m = warp_min(dtc);
      if ((threadIdx.x & 31) == 0 && m < 1.0e300)
        atomicMin(&dyn->dtmin_bits, (unsigned long long)__double_as_longlong(m));
    }
  }
}

// The FP64 momentum pass with four lanes to a particle, for simulations too
// small to fill the SMs with one (launch_momentum): lane j forms the terms of
// entry j of each list chunk, the chunk's terms change hands through shared
// memory, and each lane keeps three of the sums (j = 0: pressure gradient,
// 1: ALE1, 2: Monaghan, 3: Morris) and adds the chunk's four terms to them
// in list order, so every sum is that of the one-lane pass.  A particle's
// chain of pairs, each a chain of FP64 divisions and a square root, is what
// bounds the pass there: one lane took 31 us for the 20 neighbours of a
// 5,000-particle column.
template <int DIM, bool FUSED>
__global__ void __launch_bounds__(kSplitThreads, 4) k_momentum_split(DevBatch b) {
  chain_wait();
  constexpr int PARTS = kBlock / (kSplitThreads / 4);   // a tile's parts
  __shared__ SimDev s;
  __shared__ double terms[kSplitThreads / 4][4][13];    // [particle][entry][term]; 13: banks
  int cur = -1;
  const Particles& P = b.P;
  const unsigned FULL = 0xffffffffu;
  const int j = threadIdx.x & 3, g = threadIdx.x >> 2;
  for (int w = blockIdx.x; w < b.ntiles * PARTS; w += gridDim.x) {
    const Tile tl = b.tiles[w / PARTS];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    const int at = (w % PARTS) * (kSplitThreads / 4) + g;
    const int p = tl.start + at;
    bool active = at < tl.count && p < s.p_off + dyn->nag;
    if (FUSED && active && dyn->frozen) {
      if (j == 0) carry_record(P, p);
      active = false;
    }
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0), v4 = xi;
    double rhoi = 1.0, pi = 0.0;
    int cnt = 0;
    double wall[3] = {0, 0, 0}, tdiss[3] = {0, 0, 0}, tvisc[3] = {0, 0, 0};
    if (active) {
      xi = P.X[p];
      v4 = P.V[p];
      const double2 rp = P.RP[p];
      rhoi = rp.x;
      pi = rp.y;
      cnt = b.ncount[p];
      const int nb = P.bdt_count[p];
      if (nb > 0) {
        const double vi[3] = {v4.x, v4.y, v4.z};
        const int lam = P.L[p], bstart = P.bdt_start[p];
        if (DIM == 3) me_boundary3d(s, b, nb, bstart, vi, rhoi, pi, lam, dyn->geff, wall, tdiss, tvisc);
        else me_boundary2d(s, b, nb, bstart, vi, rhoi, pi, lam, dyn->geff, wall, tdiss, tvisc);
      }
    }
    PairSelf self;
    self.load(s, xi, v4, rhoi, pi);
    // this lane's sums; those of Morris twice, from the wall term and from 0
    double sum[3], rs[3] = {0.0, 0.0, 0.0};
    for (int d = 0; d < 3; ++d) sum[d] = j == 2 ? tdiss[d] : (j == 3 ? tvisc[d] : 0.0);
    const int nch = (cnt + 3) >> 2;
    const int nmax = __reduce_max_sync(FULL, (unsigned)nch);
    const int* list = b.nlist + 4 * list_base4(p, b.list_cap4) + j;
    // the records of the next chunk's entry are on their way while this one
    // is worked on, and the entry of the one after
    int e1 = (4 + j < cnt) ? __ldg(list + 128) : 0;
    double4 xj = xi, vj = v4;
    double2 rpj = make_double2(rhoi, pi);
    if (j < cnt) {
      const int q = __ldg(list) & kSlotMask;
      xj = load_record(P.X + q);
      vj = load_record(P.V + q);
      rpj = __ldg(P.RP + q);
    }
    for (int c = 0; c < nmax; ++c) {
      const double4 xc = xj, vc = vj;
      const double2 rc = rpj;
      const int k = 4 * c + j;
      if (k + 4 < cnt) {
        const int q = e1 & kSlotMask;
        xj = load_record(P.X + q);
        vj = load_record(P.V + q);
        rpj = __ldg(P.RP + q);
      }
      if (k + 8 < cnt) e1 = __ldg(list + (size_t)(c + 2) * 128);
      if (k < cnt) {
        double* o = terms[g][j];
        pair_terms<DIM>(s, self, xc, vc, rc,
                        [&](int kind, int d, double a) { o[3 * kind + d] = kind == 1 ? -a : a; });
      }
      __syncwarp();
      const int n = j == 3 && !self.morris ? 0 : min(cnt - 4 * c, 4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= n) break;
        const double* o = terms[g][q] + 3 * j;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          if (DIM == 2 && d == 1) continue;
          const double a = o[d];
          sum[d] = sum[d] + a;
          if (j == 3) rs[d] = rs[d] + a;
        }
      }
      __syncwarp();
    }
    // all sums to the particle's first lane
    double al[3], td[3], tv[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      al[d] = __shfl_down_sync(FULL, sum[d], 1, 4);
      td[d] = __shfl_down_sync(FULL, sum[d], 2, 4);
      tv[d] = __shfl_down_sync(FULL, sum[d], 3, 4);
      rs[d] = __shfl_down_sync(FULL, rs[d], 3, 4);
    }
    double dtc = 1.0e300;
    if (active && j == 0) {
      const double vi[3] = {v4.x, v4.y, v4.z};
      double tpres[3];
      for (int d = 0; d < 3; ++d) tpres[d] = wall[d] + sum[d] + al[d];
      momentum_close<DIM, FUSED>(s, b, dyn, p, xi, vi, rhoi, pi, tpres, td, tv, rs, dtc);
    }
    if (FUSED) {
      double m = warp_min(dtc);
      if ((threadIdx.x & 31) == 0 && m < 1.0e300)
        atomicMin(&dyn->dtmin_bits, (unsigned long long)__double_as_longlong(m));
    }
  }
}

// SASPH_continuity.f90:89-169 with AddBoundaryContribution_to_CE3D/2D: the
// wall term of drho/dt, starting value of the continuity sum (FP64).
template <int DIM>
__device__ __forceinline__ double continuity_boundary(const SimDev& s, const DevBatch& b, SimDyn* dyn, int nb,
                                                      int bstart, const double4& vi, double rhoi) {
  const Particles& P = b.P;
  double gu0 = 0, gv1 = 0, gw2 = 0;
  if (DIM == 3) {
    double gu[3] = {0, 0, 0}, gv[3] = {0, 0, 0}, gw[3] = {0, 0, 0};
    const double var[3] = {vi.x, vi.y, vi.z};
    for (int u = 0; u < nb; ++u) {
      const BdtEntry& e = P.bdt[bstart + u];
      const FaceDev& f = b.faces[s.face_off + e.clobonum - 1];
      if (!(e.loc[2] > 0.0)) continue;
      double dp = 0.0;
      for (int d = 0; d < 3; ++d) dp = dp + (2.0 * (f.velocity[d] - var[d])) * f.T[d][2];
      double dvel[3] = {dp * f.T[0][2], dp * f.T[1][2], dp * f.T[2][2]};
      double av[3];
      for (int i = 0; i < 3; ++i) {
        double a = 0.0;
        for (int k = 0; k < 3; ++k) a = a + f.T[i][k] * e.bi[3 + k];
        av[i] = a;
      }
      for (int d = 0; d < 3; ++d) {
        gu[d] = gu[d] - dvel[0] * av[d];
        gv[d] = gv[d] - dvel[1] * av[d];
        gw[d] = gw[d] - dvel[2] * av[d];
      }
    }
    gu0 = gu[0];
    gv1 = gv[1];
    gw2 = gw[2];
    atomicMax(&dyn->ncbf_max, nb);
  } else {
    const double var2[2] = {vi.x, vi.z};
    double gu_x = 0.0, gw_z = 0.0;
    for (int u = 0; u < nb; ++u) {
      const BdtEntry& e = P.bdt[bstart + u];
      const SideDev& S = b.sides[s.side_off + e.clobonum - 1];
      double IntWdS = e.bi[0];
      double dvel0, dvel1;
      if (S.zone_type == SPH_ZONE_TAPI) {
        dvel0 = 2.0 * (S.velocity[0] - var2[0]);
        dvel1 = 2.0 * (S.velocity[2] - var2[1]);
      } else {
        dvel0 = 2.0 * (-var2[0]);
        dvel1 = 2.0 * (-var2[1]);
      }
      gu_x = gu_x - dvel0 * S.nnn[0] * IntWdS;
      gw_z = gw_z - dvel1 * S.nnn[1] * IntWdS;
    }
    gu0 = gu_x;
    gw2 = gw_z;
  }
  return 0.0 - rhoi * (gu0 + gv1 + gw2);
}

// SASPH_continuity.f90:89-169 with C1_BE (3D): the frontiers complete the
// renormalisation matrices (AddBoundaryContribution_to_CE3D.f90:93-112),
// both are inverted for every particle, and with C1_divu the wall velocity
// gradients are renormalised before they enter drho/dt.
__device__ __forceinline__ double continuity_boundary_c1(const SimDev& s, const DevBatch& b, SimDyn* dyn, int nb,
                                                         int bstart, const double4& vi, double rhoi, int p) {
  const Particles& P = b.P;
  const int total = P.total_slots;
  const bool divu = s.c1_divu != 0;
  double Bg[9], Bd[9];
  load_b(P.BG, total, p, Bg);
  if (divu) load_b(P.BD, total, p, Bd);
  double gu[3] = {0, 0, 0}, gv[3] = {0, 0, 0}, gw[3] = {0, 0, 0};
  const double var[3] = {vi.x, vi.y, vi.z};
  for (int u = 0; u < nb; ++u) {
    const BdtEntry& e = P.bdt[bstart + u];
    const FaceDev& f = b.faces[s.face_off + e.clobonum - 1];
    if (!(e.loc[2] > 0.0)) continue;
    if (divu) add_frontier_b(f, e, Bd);
    add_frontier_b(f, e, Bg);
    double dp = 0.0;
    for (int d = 0; d < 3; ++d) dp = dp + (2.0 * (f.velocity[d] - var[d])) * f.T[d][2];
    double dvel[3] = {dp * f.T[0][2], dp * f.T[1][2], dp * f.T[2][2]};
    double av[3];
    for (int i = 0; i < 3; ++i) {
      double a = 0.0;
      for (int k = 0; k < 3; ++k) a = a + f.T[i][k] * e.bi[3 + k];
      av[i] = a;
    }
    for (int d = 0; d < 3; ++d) {
      gu[d] = gu[d] - dvel[0] * av[d];
      gv[d] = gv[d] - dvel[1] * av[d];
      gw[d] = gw[d] - dvel[2] * av[d];
    }
  }
  if (divu) b_inversion(Bd, s.invb_det_thresh);
  b_inversion(Bg, s.invb_det_thresh);
  store_b(P.BG, total, p, Bg);
  if (divu) store_b(P.BD, total, p, Bd);
  if (nb == 0) return 0.0;
  atomicMax(&dyn->ncbf_max, nb);
  if (divu) {
    b_renormalise(Bd, gu);
    b_renormalise(Bd, gv);
    b_renormalise(Bd, gw);
  }
  return 0.0 - rhoi * (gu[0] + gv[1] + gw[2]);
}

// One pair's three terms of the velocity divergence (Continuity_Equation.f90).
template <int DIM>
__device__ __forceinline__ void continuity_terms(const SimDev& s, const double4& xi, const double4& vi, double rhoi,
                                                 const double4& xj, const double4& vj, double* T) {
  double r0 = xi.x - xj.x, r1 = xi.y - xj.y, r2 = xi.z - xj.z;
  double rr = r0 * r0 + r1 * r1 + r2 * r2;
  double PK1, PK2, PK3;
  kernel_values(s, rr, PK1, PK2, PK3);
  double c = rhoi * vj.w * PK1;     // rhoi * (amassj / rhoj) * PK1
  T[0] = c * (vj.x - vi.x) * r0;
  if (DIM == 3) T[1] = c * (vj.y - vi.y) * r1;
  T[2] = c * (vj.z - vi.z) * r2;
}

// drho/dt of particle p; in the fused step Leapfrog_continuity.f90:54-68 and
// EoS_barotropic_linear.f90:49-55.
template <bool FUSED>
__device__ __forceinline__ void continuity_close(const SimDev& s, const DevBatch& b, const SimDyn* dyn, int p,
                                                 double rhoi, double dden) {
  if (FUSED) {
    double rho = rhoi + dyn->dt * dden;
    if (s.density_thresholds == 1) {
      if (rho < 0.9 * s.den0) rho = 0.9 * s.den0;
      if (rho > 1.1 * s.den0) rho = 1.1 * s.den0;
    }
    double pr = s.k_over_rho0 * (rho - s.den0) + s.p_ref;
    b.P.RP[p] = make_double2(rho, pr);
  } else {
    b.P.DDEN[p] = dden;
  }
}

// Continuity, FP64 form: SASPH_continuity + Continuity_Equation, optionally
// fused with Leapfrog_continuity and the EoS.  C1 (3D): the renormalised
// form, Continuity_Equation.f90:119-126,201-217 -- the whole velocity
// gradient vectors are summed, and renormalised with B_ren_divu when
// C1_divu is set; their trace equals the plain form's sum bit for bit.
// BATCH (not with C1): two list entries' records requested before the
// first one's arithmetic, as in k_momentum; the same sums.
template <int DIM, bool FUSED, bool C1 = false, bool BATCH = false>
__global__ void __launch_bounds__(kBlock, 2) k_continuity(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !(FUSED && dyn->frozen);
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    double4 vi = make_double4(0.0, 0.0, 0.0, 0.0);
    double rhoi = 1.0, dden = 0.0;
    int cnt = 0;
    if (active) {
      xi = P.X[p];
      vi = P.V[p];
      rhoi = P.RP[p].x;
      cnt = b.ncount[p];
      int nb = P.bdt_count[p];
      if (C1 && s.c1_be) dden = continuity_boundary_c1(s, b, dyn, nb, nb > 0 ? P.bdt_start[p] : 0, vi, rhoi, p);
      else if (nb > 0) dden = continuity_boundary<DIM>(s, b, dyn, nb, P.bdt_start[p], vi, rhoi);
    }
    double a1 = 0.0, a2 = 0.0, a3 = 0.0;
    double g1[3] = {0, 0, 0}, g2[3] = {0, 0, 0}, g3[3] = {0, 0, 0};
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    auto pair = [&](const double4& xj, const double4& vj) {
      if (C1) {
        double r0 = xi.x - xj.x, r1 = xi.y - xj.y, r2 = xi.z - xj.z;
        double rr = r0 * r0 + r1 * r1 + r2 * r2;
        double PK1, PK2, PK3;
        kernel_values(s, rr, PK1, PK2, PK3);
        double c = rhoi * vj.w * PK1;     // rhoi * (amassj / rhoj) * PK1
        const double c0 = c * (vj.x - vi.x), c1 = c * (vj.y - vi.y), c2 = c * (vj.z - vi.z);
        g1[0] = g1[0] + c0 * r0;
        g1[1] = g1[1] + c0 * r1;
        g1[2] = g1[2] + c0 * r2;
        g2[0] = g2[0] + c1 * r0;
        g2[1] = g2[1] + c1 * r1;
        g2[2] = g2[2] + c1 * r2;
        g3[0] = g3[0] + c2 * r0;
        g3[1] = g3[1] + c2 * r1;
        g3[2] = g3[2] + c2 * r2;
      } else {
        double T[3];
        continuity_terms<DIM>(s, xi, vi, rhoi, xj, vj, T);
        a1 = a1 + T[0];
        if (DIM == 3) a2 = a2 + T[1];
        a3 = a3 + T[2];
      }
    };
    if (BATCH) {
      for (int k = 0; k < nmax; k += 2) {
        const int e0 = lr.get(k);
        const int e1 = k + 1 < nmax ? lr.get(k + 1) : 0;
        const bool u0 = k < cnt, u1 = k + 1 < cnt;
        double4 x0 = make_double4(0.0, 0.0, 0.0, 0.0), v0 = x0, x1 = x0, v1 = x0;
        if (u0) {
          const int q = e0 & kSlotMask;
          x0 = load_record(P.X + q); v0 = load_record(P.V + q);
        }
        if (u1) {
          const int q = e1 & kSlotMask;
          x1 = load_record(P.X + q); v1 = load_record(P.V + q);
        }
        if (u0) pair(x0, v0);
        if (u1) pair(x1, v1);
      }
    } else {
      for (int k = 0; k < nmax; ++k) {
        int e = lr.get(k);
        if (k >= cnt) continue;
        int q = e & kSlotMask;
        pair(load_record(P.X + q), load_record(P.V + q));
      }
    }
    if (active) {
      if (C1) {
        if (s.c1_be && s.c1_divu) {
          double B[9];
          load_b(P.BD, P.total_slots, p, B);
          b_renormalise(B, g1);
          b_renormalise(B, g2);
          b_renormalise(B, g3);
        }
        dden = dden - (g1[0] + g2[1] + g3[2]);
      } else if (DIM == 3) {
        dden = dden - (a1 + a2 + a3);
      } else {
        dden = dden - (a1 + a3);
      }
      continuity_close<FUSED>(s, b, dyn, p, rhoi, dden);
    }
  }
}

// The FP64 continuity pass with four lanes to a particle (k_momentum_split's
// scheme): lane d keeps the sum of component d.
template <int DIM, bool FUSED>
__global__ void __launch_bounds__(kSplitThreads, 4) k_continuity_split(DevBatch b) {
  chain_wait();
  constexpr int PARTS = kBlock / (kSplitThreads / 4);
  __shared__ SimDev s;
  __shared__ double terms[kSplitThreads / 4][4][3];
  int cur = -1;
  const Particles& P = b.P;
  const unsigned FULL = 0xffffffffu;
  const int j = threadIdx.x & 3, g = threadIdx.x >> 2;
  for (int w = blockIdx.x; w < b.ntiles * PARTS; w += gridDim.x) {
    const Tile tl = b.tiles[w / PARTS];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    const int at = (w % PARTS) * (kSplitThreads / 4) + g;
    const int p = tl.start + at;
    const bool active = at < tl.count && p < s.p_off + dyn->nag && !(FUSED && dyn->frozen);
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0), vi = xi;
    double rhoi = 1.0;
    int cnt = 0;
    if (active) {
      xi = P.X[p];
      vi = P.V[p];
      rhoi = P.RP[p].x;
      cnt = b.ncount[p];
    }
    double sum = 0.0;
    const int nch = (cnt + 3) >> 2;
    const int nmax = __reduce_max_sync(FULL, (unsigned)nch);
    const int* list = b.nlist + 4 * list_base4(p, b.list_cap4) + j;
    int e1 = (4 + j < cnt) ? __ldg(list + 128) : 0;
    double4 xj = xi, vj = vi;
    if (j < cnt) {
      const int q = __ldg(list) & kSlotMask;
      xj = load_record(P.X + q);
      vj = load_record(P.V + q);
    }
    for (int c = 0; c < nmax; ++c) {
      const double4 xc = xj, vc = vj;
      const int k = 4 * c + j;
      if (k + 4 < cnt) {
        const int q = e1 & kSlotMask;
        xj = load_record(P.X + q);
        vj = load_record(P.V + q);
      }
      if (k + 8 < cnt) e1 = __ldg(list + (size_t)(c + 2) * 128);
      if (k < cnt) continuity_terms<DIM>(s, xi, vi, rhoi, xc, vc, terms[g][j]);
      __syncwarp();
      const int n = (j == 3 || (DIM == 2 && j == 1)) ? 0 : min(cnt - 4 * c, 4);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= n) break;
        sum = sum + terms[g][q][j];
      }
      __syncwarp();
    }
    const double a2 = __shfl_down_sync(FULL, sum, 1, 4), a3 = __shfl_down_sync(FULL, sum, 2, 4);
    if (active && j == 0) {
      const int nb = P.bdt_count[p];
      double dden = 0.0;
      if (nb > 0) dden = continuity_boundary<DIM>(s, b, dyn, nb, P.bdt_start[p], vi, rhoi);
      if (DIM == 3) dden = dden - (sum + a2 + a3);
      else dden = dden - (sum + a3);
      continuity_close<FUSED>(s, b, dyn, p, rhoi, dden);
    }
  }
}

// ==========================================================================
// FP32-compensated form.  Pair arithmetic in FP32 on the screening copies
// (FP64 cell origin + FP32 offset) with compensated (Kahan) per-particle
// sums; the pressure term uses the symmetric form that the two accumulators
// of inter_EqMoto.f90:195-221 add up to.  Boundary terms, the elastic
// reaction, time integration and the time step stay in FP64.
// ==========================================================================
struct Kahan {
  float s, c;
  __device__ __forceinline__ void zero() {
    s = 0.f;
    c = 0.f;
  }
  // built without contraction (--fmad=false), as compensation requires
  __device__ __forceinline__ void add(float x) {
    float y = x - c;
    float t = s + y;
    c = (t - s) - y;
    s = t;
  }
  __device__ __forceinline__ double val() const { return (double)s - (double)c; }
};

struct F32Const {
  float hinv, h2inv, eta, eta2, ke, kacl, amon, nu, nu4;
  __device__ __forceinline__ void load(const SimDev& s) {
    hinv = (float)(1.0 / s.h);
    h2inv = (float)(1.0 / s.squareh);
    eta = (float)s.eta;
    eta2 = (float)s.eta2;
    ke = (float)s.ke_coef;
    kacl = (float)s.kacl_coef;
    amon = (float)(s.alfa_mon * (s.celerita + s.celerita) * s.h);
    nu = (float)s.kin_visc;
    nu4 = (float)(4.0 * (s.kin_visc * s.kin_visc));
  }
};

// The PTX approximate reciprocal and reciprocal square root (one special
// function unit instruction each, relative error about 2^-23, subnormals
// flushed): the FP32c pair terms' divisions and square roots.
__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Distance of a list pair from its squared distance: rr is positive for any
// two particles of distinct positions; the floor keeps r finite (0) should
// two FP32 offsets coincide.
__device__ __forceinline__ float pair_distance(float rr) {
  const float rq = fmaxf(rr, 1.0e-30f);
  return rq * rsqrt_approx(rq);
}

// Beta-spline gradient factors of a list pair (CalcVarLength.f90:230-262):
// PK1 = g ke / (r + eta), PK2 = PK1 / (rr + eta2), PK3 = gw kacl / (r + eta).
// The two divisions share one reciprocal: 1/a = b/(ab), 1/b = a/(ab).  A
// list pair has r <= 2h in FP64; its FP32 q may round a hair past 2, where
// both polynomials vanish to within rounding, so no support test is needed.
__device__ __forceinline__ void kernel_values_f32(const F32Const& c, float rr, float& PK1, float& PK2, float& PK3) {
  const float r = pair_distance(rr);
  const float q = r * c.hinv;
  const float q2 = rr * c.h2inv;
  const float a = r + c.eta, bq = rr + c.eta2;
  const float inv = rcp_approx(a * bq);
  const float denom = bq * inv;
  const float g = (q < 1.0f) ? fmaf(1.5f, q2, -2.0f * q) : fmaf(-0.5f, q2, fmaf(2.0f, q, -2.0f));
  const float gw = fmaf(12.0f, q, fmaf(-3.0f, q2, -12.0f));
  PK1 = g * c.ke * denom;
  PK2 = PK1 * (a * inv);
  PK3 = gw * c.kacl * denom;
}

// PK1 alone (the continuity pass).
__device__ __forceinline__ float kernel_pk1_f32(const F32Const& c, float rr) {
  const float r = pair_distance(rr);
  const float q = r * c.hinv;
  const float q2 = rr * c.h2inv;
  const float g = (q < 1.0f) ? fmaf(1.5f, q2, -2.0f * q) : fmaf(-0.5f, q2, fmaf(2.0f, q, -2.0f));
  return g * c.ke * rcp_approx(r + c.eta);
}

// Cell-origin offset of the neighbour column (run) a list entry names.  A
// lane's entries are stored run by run, so the offsets are formed again only
// when the run changes: (ci - ir) dcd = (1 - rx) dcd for the run's x column
// rx = r % 3 (r in 2D) and likewise in y.
template <int DIM>
struct RunCursor {
  int r = -1;
  float Dx = 0.f, Dy = 0.f;
  __device__ __forceinline__ void update(const SimDev& s, int run) {
    if (run == r) return;
    r = run;
    const int rx = (DIM == 3) ? run % 3 : run;
    Dx = (float)(1 - rx) * s.dcdf[0];
    Dy = (DIM == 3) ? (float)(1 - run / 3) * s.dcdf[1] : 0.f;
  }
};

// FP32 separation x_i - x_j of list entry e with neighbour record xj: the
// cell-origin difference (run offsets in x and y, (k_i - k_j) dcd in z, all
// exact small multiples) plus the offsets' difference.
template <int DIM>
__device__ __forceinline__ void separation_f32(const SimDev& s, RunCursor<DIM>& rc, int e, const float4& xj,
                                               const float4& xfi, float ckf, float dz, float& d0, float& d1,
                                               float& d2) {
  rc.update(s, (int)((unsigned)e >> kSlotBits));
  d0 = rc.Dx + (xfi.x - xj.x);
  d1 = (DIM == 3) ? rc.Dy + (xfi.y - xj.y) : 0.f;
  d2 = (ckf - xj.w) * dz + (xfi.z - xj.z);
}

// The closing of an FP32c momentum pass for particle p, from its nine pair
// sums ms and its FP64 wall terms (zero without close faces): the laminar
// flag (inter_EqMoto.f90:269-283), gravity, the elastic reaction, and in
// the fused step the leapfrog update and the particle's CFL time.  One
// function for both places a particle is closed (the finishing launch, and
// the pair launch itself for particles without close faces), so the two
// give the same bits.
template <int DIM, bool FUSED>
__device__ __forceinline__ void momentum_f32_close(const SimDev& s, const DevBatch& b, SimDyn* dyn, int p,
                                                   const double* ms, double* tpres, const double* tdiss,
                                                   const double* tvisc, const double* vi, double rhoi, double pi,
                                                   int nb, int bstart, double& dtc) {
  const Particles& P = b.P;
  const double GI = (double)9.80665f;   // Static_allocation_module.f90:72, a default-REAL literal
  const double* geff = dyn->geff;
  double rs0 = ms[6], rs1 = ms[7], rs2 = ms[8];
  tpres[0] = tpres[0] + ms[0];
  tpres[1] = tpres[1] + ms[1];
  tpres[2] = tpres[2] + ms[2];
  int lam_new = 0;
  if (s.kin_visc > 0.0) {
    double absv_pres = sqrt(tpres[0] * tpres[0] + tpres[1] * tpres[1] + tpres[2] * tpres[2]) + GI;
    double absv_morris = sqrt(rs0 * rs0 + rs1 * rs1 + rs2 * rs2);
    double weight = 0.0;
    if (absv_pres != 0.0) weight = absv_morris / absv_pres * 100.0;
    lam_new = (weight > 5.0 || absv_pres == 0.0) ? 1 : 0;
  }
  double acc[3];
  acc[0] = tpres[0] + (tdiss[0] + ms[3]) + (tvisc[0] + rs0) + geff[0];
  acc[1] = tpres[1] + (tdiss[1] + ms[4]) + (tvisc[1] + rs1) + geff[1];
  acc[2] = tpres[2] + (tdiss[2] + ms[5]) + (tvisc[2] + rs2) + geff[2];
  const double4 xi = P.X[p];
  if (nb > 0) {
    double R[3];
    const double xa[3] = {xi.x, xi.y, xi.z};
    elastic_reaction<DIM>(s, b, nb, bstart, xa, vi, R);
    for (int d = 0; d < 3; ++d) acc[d] = acc[d] + R[d];
  }
  if (FUSED) {
    double dtvel = dyn->dtvel, dt = dyn->dt;
    double vn[3];
    for (int d = 0; d < 3; ++d) vn[d] = vi[d] + dtvel * acc[d];
    P.X2[p] = make_double4(xi.x + dt * vn[0], xi.y + dt * vn[1], xi.z + dt * vn[2], xi.w);
    P.V2[p] = make_double4(vn[0], vn[1], vn[2], rhoi);
    if (P.VF2) P.VF2[p] = make_float4((float)vn[0], (float)vn[1], (float)vn[2], 0.f);
    P.P2[p] = pi;
    P.I2[p] = P.I[p];
    P.L2[p] = (uint8_t)lam_new;
    double U = sqrt(vn[0] * vn[0] + vn[1] * vn[1] + vn[2] * vn[2]);
    // with velocity smoothing the CFL minimum is taken on the smoothed
    // velocities (k_velocity_smoothing_apply), which also moves X2
    if (!(s.teta_v > 1.0e-9)) dtc = s.cfl * 2.0 * s.h / (s.celerita + U);
  } else {
    P.ACC[p] = make_double4(acc[0], acc[1], acc[2], 0.0);
    P.L[p] = (uint8_t)lam_new;
  }
}

// A particle's FP32c momentum pairs: its own values and the sums of the list
// chunk at hand.
template <int DIM, bool C1>
struct MomentumPairs {
  const SimDev& s;
  const double2* __restrict__ rp;   // (C1) densities and pressures
  F32Const fc;
  RunCursor<DIM> rc;
  float4 xfi;
  float ckf, dz, vix, viy, viz, rhof, Pi;
  double piD;
  bool morris;
  float cp0, cp1, cp2, cd0, cd1, cd2, cv0, cv1, cv2, cg0, cg1, cg2;
  __device__ __forceinline__ MomentumPairs(const SimDev& sim, const double2* r) : s(sim), rp(r) {
    fc.load(sim);
    xfi = make_float4(0.f, 0.f, 0.f, 0.f);
    vix = viy = viz = Pi = ckf = 0.f;
    rhof = 1.f;
    piD = 0.0;
    dz = sim.dcdf[2];
    morris = sim.kin_visc > 1.0e-12;
    clear();
  }
  __device__ __forceinline__ void load(const float4& x, const double4& v, const double2& r) {
    xfi = x;
    ckf = x.w;
    vix = (float)v.x;
    viy = (float)v.y;
    viz = (float)v.z;
    rhof = (float)r.x;
    Pi = (float)(r.y / (r.x * r.x));
    piD = r.y;
  }
  __device__ __forceinline__ void clear() {
    cp0 = cp1 = cp2 = cd0 = cd1 = cd2 = cv0 = cv1 = cv2 = 0.f;
    if (C1) cg0 = cg1 = cg2 = 0.f;
  }
  // a neighbour's record is 40 B: XF (offset, cell k), VF (velocity,
  // m/rho) and RM (rho, p/rho^2); its mass is rho (m/rho)
  __device__ __forceinline__ void pair(int e, const float4& xj, const float4& vj, const float2& rmj) {
    const int q = e & kSlotMask;
    float d0, d1, d2;
    separation_f32<DIM>(s, rc, e, xj, xfi, ckf, dz, d0, d1, d2);
    float rr = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
    float PK1, PK2, PK3;
    kernel_values_f32(fc, rr, PK1, PK2, PK3);
    const float rhoj = rmj.x;
    const float mj = rhoj * vj.w;
    // pressure (both accumulators of inter_EqMoto together)
    float pf = -(mj * (Pi + rmj.y) * PK3);
    cp0 = fmaf(pf, d0, cp0);
    if (DIM == 3) cp1 = fmaf(pf, d1, cp1);
    cp2 = fmaf(pf, d2, cp2);
    if (C1) {
      const float dpf = (float)(__ldg(reinterpret_cast<const double*>(rp + q) + 1) - piD);
      const float gf = -(mj * dpf * rcp_approx(rhof * rhoj) * PK3);
      cg0 = fmaf(gf, d0, cg0);
      if (DIM == 3) cg1 = fmaf(gf, d1, cg1);
      cg2 = fmaf(gf, d2, cg2);
    }
    float dv0 = vj.x - vix, dv1 = vj.y - viy, dv2 = vj.z - viz;
    // viscomon amon / rsum and viscomorris nu4 / (nu rsum + 1e-3) from one
    // reciprocal of their denominators' product
    const float rsum = rhof + rhoj;
    const float bm = fmaf(fc.nu, rsum, 1.0e-3f);
    const float iv = rcp_approx(rsum * bm);
    float vr = -fmaf(dv2, d2, fmaf(dv1, d1, dv0 * d0));
    float df = mj * (fc.amon * (bm * iv)) * vr * PK2;
    cd0 = fmaf(df, d0, cd0);
    if (DIM == 3) cd1 = fmaf(df, d1, cd1);
    cd2 = fmaf(df, d2, cd2);
    if (morris) {
      float vf = -((mj * fc.nu4) * (rsum * iv) * PK2 * rr);
      cv0 = fmaf(vf, dv0, cv0);
      if (DIM == 3) cv1 = fmaf(vf, dv1, cv1);
      cv2 = fmaf(vf, dv2, cv2);
    }
  }
  // `pair` for entries ea, eb on paired instructions: every half rounds as
  // the scalar instruction does (x - y as fma(y, -1, x), one rounding
  // either way; products and sums in the scalar code's association, no
  // contraction), the special-function values, the cubic spline's branch
  // and the accumulations stay scalar, ea's accumulated before eb's.
  __device__ __forceinline__ void pair2(int ea, int eb, const float4& xa, const float4& va, const float2& ra,
                                        const float4& xb, const float4& vb, const float2& rb) {
    const float2 m1 = make_float2(-1.f, -1.f);
    rc.update(s, (int)((unsigned)ea >> kSlotBits));
    const float dxa = rc.Dx, dya = rc.Dy;
    rc.update(s, (int)((unsigned)eb >> kSlotBits));
    const float2 Dx = make_float2(dxa, rc.Dx), Dy = make_float2(dya, rc.Dy);
    const float2 d0 = __fadd2_rn(Dx, __ffma2_rn(make_float2(xa.x, xb.x), m1, make_float2(xfi.x, xfi.x)));
    const float2 d1 = (DIM == 3) ? __fadd2_rn(Dy, __ffma2_rn(make_float2(xa.y, xb.y), m1, make_float2(xfi.y, xfi.y)))
                                 : make_float2(0.f, 0.f);
    const float2 dk = __ffma2_rn(make_float2(xa.w, xb.w), m1, make_float2(ckf, ckf));
    const float2 d2 = __fadd2_rn(__fmul2_rn(dk, make_float2(dz, dz)),
                                 __ffma2_rn(make_float2(xa.z, xb.z), m1, make_float2(xfi.z, xfi.z)));
    const float2 rr = __ffma2_rn(d2, d2, __ffma2_rn(d1, d1, __fmul2_rn(d0, d0)));
    // kernel_values_f32
    const float2 rq = make_float2(fmaxf(rr.x, 1.0e-30f), fmaxf(rr.y, 1.0e-30f));
    const float2 r = __fmul2_rn(rq, make_float2(rsqrt_approx(rq.x), rsqrt_approx(rq.y)));
    const float2 q = __fmul2_rn(r, make_float2(fc.hinv, fc.hinv));
    const float2 q2 = __fmul2_rn(rr, make_float2(fc.h2inv, fc.h2inv));
    const float2 a = __fadd2_rn(r, make_float2(fc.eta, fc.eta));
    const float2 bq = __fadd2_rn(rr, make_float2(fc.eta2, fc.eta2));
    const float2 ab = __fmul2_rn(a, bq);
    const float2 inv = make_float2(rcp_approx(ab.x), rcp_approx(ab.y));
    const float2 denom = __fmul2_rn(bq, inv);
    const float2 glo = __ffma2_rn(make_float2(1.5f, 1.5f), q2, __fmul2_rn(make_float2(-2.0f, -2.0f), q));
    const float2 ghi = __ffma2_rn(make_float2(-0.5f, -0.5f), q2,
                                  __ffma2_rn(make_float2(2.0f, 2.0f), q, make_float2(-2.0f, -2.0f)));
    const float2 g = make_float2(q.x < 1.0f ? glo.x : ghi.x, q.y < 1.0f ? glo.y : ghi.y);
    const float2 gw = __ffma2_rn(make_float2(12.0f, 12.0f), q,
                                 __ffma2_rn(make_float2(-3.0f, -3.0f), q2, make_float2(-12.0f, -12.0f)));
    const float2 PK1 = __fmul2_rn(__fmul2_rn(g, make_float2(fc.ke, fc.ke)), denom);
    const float2 PK2 = __fmul2_rn(PK1, __fmul2_rn(a, inv));
    const float2 PK3 = __fmul2_rn(__fmul2_rn(gw, make_float2(fc.kacl, fc.kacl)), denom);
    const float2 mj = __fmul2_rn(make_float2(ra.x, rb.x), make_float2(va.w, vb.w));
    // pressure: pf = -t
    const float2 t = __fmul2_rn(__fmul2_rn(mj, __fadd2_rn(make_float2(Pi, Pi), make_float2(ra.y, rb.y))), PK3);
    // viscosity
    const float2 dv0 = __ffma2_rn(make_float2(vix, vix), m1, make_float2(va.x, vb.x));
    const float2 dv1 = __ffma2_rn(make_float2(viy, viy), m1, make_float2(va.y, vb.y));
    const float2 dv2 = __ffma2_rn(make_float2(viz, viz), m1, make_float2(va.z, vb.z));
    const float2 rsum = __fadd2_rn(make_float2(rhof, rhof), make_float2(ra.x, rb.x));
    const float2 bm = __ffma2_rn(make_float2(fc.nu, fc.nu), rsum, make_float2(1.0e-3f, 1.0e-3f));
    const float2 rb2 = __fmul2_rn(rsum, bm);
    const float2 iv = make_float2(rcp_approx(rb2.x), rcp_approx(rb2.y));
    // vr = -u; df = -w
    const float2 u = __ffma2_rn(dv2, d2, __ffma2_rn(dv1, d1, __fmul2_rn(dv0, d0)));
    const float2 w = __fmul2_rn(
        __fmul2_rn(__fmul2_rn(mj, __fmul2_rn(make_float2(fc.amon, fc.amon), __fmul2_rn(bm, iv))), u), PK2);
    cp0 = fmaf(-t.x, d0.x, cp0);
    if (DIM == 3) cp1 = fmaf(-t.x, d1.x, cp1);
    cp2 = fmaf(-t.x, d2.x, cp2);
    cd0 = fmaf(-w.x, d0.x, cd0);
    if (DIM == 3) cd1 = fmaf(-w.x, d1.x, cd1);
    cd2 = fmaf(-w.x, d2.x, cd2);
    cp0 = fmaf(-t.y, d0.y, cp0);
    if (DIM == 3) cp1 = fmaf(-t.y, d1.y, cp1);
    cp2 = fmaf(-t.y, d2.y, cp2);
    cd0 = fmaf(-w.y, d0.y, cd0);
    if (DIM == 3) cd1 = fmaf(-w.y, d1.y, cd1);
    cd2 = fmaf(-w.y, d2.y, cd2);
    if (morris) {
      // vf = -z
      const float2 z = __fmul2_rn(
          __fmul2_rn(__fmul2_rn(__fmul2_rn(mj, make_float2(fc.nu4, fc.nu4)), __fmul2_rn(rsum, iv)), PK2), rr);
      cv0 = fmaf(-z.x, dv0.x, cv0);
      if (DIM == 3) cv1 = fmaf(-z.x, dv1.x, cv1);
      cv2 = fmaf(-z.x, dv2.x, cv2);
      cv0 = fmaf(-z.y, dv0.y, cv0);
      if (DIM == 3) cv1 = fmaf(-z.y, dv1.y, cv1);
      cv2 = fmaf(-z.y, dv2.y, cv2);
    }
  }
  // the entries of a chunk, rem of them, their records requested together
  template <bool PAIRED>
  __device__ __forceinline__ void chunk(const Particles& P, const int4& ch, int rem) {
    float4 x0, v0, x1, v1, x2, v2, x3, v3;
    float2 r0, r1, r2, r3;
    const int q0 = ch.x & kSlotMask, q1 = ch.y & kSlotMask, q2 = ch.z & kSlotMask, q3 = ch.w & kSlotMask;
    x0 = __ldg(P.XF + q0); v0 = __ldg(P.VF + q0); r0 = __ldg(P.RM + q0);
    if (rem > 1) { x1 = __ldg(P.XF + q1); v1 = __ldg(P.VF + q1); r1 = __ldg(P.RM + q1); }
    if (rem > 2) { x2 = __ldg(P.XF + q2); v2 = __ldg(P.VF + q2); r2 = __ldg(P.RM + q2); }
    if (rem > 3) { x3 = __ldg(P.XF + q3); v3 = __ldg(P.VF + q3); r3 = __ldg(P.RM + q3); }
    if (PAIRED) {
      if (rem > 1) pair2(ch.x, ch.y, x0, v0, r0, x1, v1, r1);
      else pair(ch.x, x0, v0, r0);
      if (rem > 3) pair2(ch.z, ch.w, x2, v2, r2, x3, v3, r3);
      else if (rem > 2) pair(ch.z, x2, v2, r2);
    } else {
      pair(ch.x, x0, v0, r0);
      if (rem > 1) pair(ch.y, x1, v1, r1);
      if (rem > 2) pair(ch.z, x2, v2, r2);
      if (rem > 3) pair(ch.w, x3, v3, r3);
    }
  }
};

// Momentum, FP32c form, in two launches.  k_momentum_f32 holds only what
// the pair loop needs -- the particle's FP32 values, the compensated sums,
// the list chunk being read and the next one -- so that it runs at 3 blocks
// of 256 per SM with 12 bytes a thread spilled (gathers are latency-bound:
// occupancy pays more than loading the next pair's records ahead), and writes the nine
// compensated sums of each particle to MSUM.
// k_momentum_f32_finish adds the FP64 wall terms (an independent sum), the
// laminar flag, gravity and the elastic reaction and, in the fused step,
// the leapfrog update and the CFL minimum.
// C1 (C1_BE): the pressure-gradient accumulator of inter_EqMoto.f90:195-204,
// -m_j (p_j - p_i) / (rho_i rho_j) PK3 r, is summed apart as well (the
// pressure difference formed in FP64), so the finishing launch can
// renormalise it with B_ren_gradp (inter_EqMoto.f90:255-260) and keep the
// ALE1 accumulator, the symmetric sum less it, as it is.
// BATCH: the twelve neighbour records of a list chunk are all requested
// before the first pair's arithmetic, four pairs' loads in flight per lane
// instead of one, at 2 blocks of 256 per SM (the registers they need); the
// autotuner chooses it or the lean loop (3 blocks per SM) on the live
// state.  Both sum the same terms in the same order: identical results.
// fused (the whole step, not C1): a particle without close faces has no
// FP64 wall terms, so this launch closes it at once (momentum_f32_close,
// the finishing launch's own code) instead of passing its nine sums on.
// PAIRED (with BATCH, not C1): two list entries' terms on Blackwell's paired
// FP32 instructions (pair2), the same bits as two calls of `pair`.
template <int DIM, bool C1 = false, bool BATCH = false, bool PAIRED = false>
__global__ void __launch_bounds__(kBlock, (C1 || BATCH) ? 2 : 3) k_momentum_f32(DevBatch b, int fused) {
  chain_wait();
  static_assert(!PAIRED || (BATCH && !C1), "the paired loop is a batched, non-C1 shape");
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    const bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen;
    int cnt = 0;
    MomentumPairs<DIM, C1> m(s, P.RP);
    if (active) {
      m.load(P.XF[p], P.V[p], P.RP[p]);
      cnt = b.ncount[p];
    }
    // compensated sums of 4-entry partial sums (one list chunk each)
    Kahan tp0, tp1, tp2, td0, td1, td2, tv0, tv1, tv2;
    tp0.zero(); tp1.zero(); tp2.zero(); td0.zero(); td1.zero(); td2.zero(); tv0.zero(); tv1.zero(); tv2.zero();
    Kahan tg0, tg1, tg2;
    tg0.zero(); tg1.zero(); tg2.zero();
    // one list chunk (4 entries) per iteration: entries, compensation and
    // the next chunk's load handled once per chunk
    const int nch = (cnt + 3) >> 2;
    const int nchmax = __reduce_max_sync(0xffffffffu, (unsigned)nch);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nchmax * 4);
    const int4* lbase = reinterpret_cast<const int4*>(b.nlist) + list_base4(p, b.list_cap4);
    int4 nxt = nch > 0 ? __ldg(lbase) : make_int4(0, 0, 0, 0);
    for (int c = 0; c < nchmax; ++c) {
      const int4 ch = nxt;
      if (c + 1 < nch) nxt = __ldg(lbase + (size_t)(c + 1) * 32);
      if (c >= nch) continue;
      const int rem = cnt - 4 * c;   // >= 1
      if (BATCH) {
        m.template chunk<PAIRED>(P, ch, rem);
      } else {
        auto one = [&](int e) {
          const int q = e & kSlotMask;
          m.pair(e, __ldg(P.XF + q), __ldg(P.VF + q), __ldg(P.RM + q));
        };
        one(ch.x);
        if (rem > 1) one(ch.y);
        if (rem > 2) one(ch.z);
        if (rem > 3) one(ch.w);
      }
      tp0.add(m.cp0); tp1.add(m.cp1); tp2.add(m.cp2);
      td0.add(m.cd0); td1.add(m.cd1); td2.add(m.cd2);
      tv0.add(m.cv0); tv1.add(m.cv1); tv2.add(m.cv2);
      if (C1) {
        tg0.add(m.cg0); tg1.add(m.cg1); tg2.add(m.cg2);
      }
      m.clear();
    }
    bool close_here = false;
    if (!C1 && fused && active) close_here = P.bdt_count[p] == 0;
    double dtc = 1.0e300;
    if (close_here) {
      const double ms[9] = {tp0.val(), tp1.val(), tp2.val(), td0.val(), td1.val(), td2.val(),
                            tv0.val(), tv1.val(), tv2.val()};
      double tpres[3] = {0, 0, 0};
      const double tdiss[3] = {0, 0, 0}, tvisc[3] = {0, 0, 0};
      const double4 v4 = P.V[p];
      const double2 rp = P.RP[p];
      const double vi[3] = {v4.x, v4.y, v4.z};
      momentum_f32_close<DIM, true>(s, b, dyn, p, ms, tpres, tdiss, tvisc, vi, rp.x, rp.y, 0, 0, dtc);
    }
    if (!C1 && fused) {
      const double least = warp_min(dtc);
      if ((threadIdx.x & 31) == 0 && least < 1.0e300)
        atomicMin(&dyn->dtmin_bits, (unsigned long long)__double_as_longlong(least));
    }
    if (active && !close_here) {
      double* o = P.MSUM + p;
      const size_t st = (size_t)P.total_slots;   // component-major: coalesced
      o[0] = tp0.val();
      o[st] = tp1.val();
      o[2 * st] = tp2.val();
      o[3 * st] = td0.val();
      o[4 * st] = td1.val();
      o[5 * st] = td2.val();
      o[6 * st] = tv0.val();
      o[7 * st] = tv1.val();
      o[8 * st] = tv2.val();
      if (C1) {
        o[9 * st] = tg0.val();
        o[10 * st] = tg1.val();
        o[11 * st] = tg2.val();
      }
    }
  }
}

// k_momentum_f32 with four lanes to a particle, for simulations too small to
// fill the SMs with one (momentum_split): lane j of a particle sums list
// chunks j, j + 4, ... and the chunk sums change hands through shared
// memory; lane j < 3 keeps the compensated sums of one kind (pressure,
// Monaghan, Morris) and adds the chunks to them in list order, so every sum
// is that of the one-lane pass.  Lanes 8 j .. 8 j + 7 of a warp hold lane j of
// its eight particles: neighbouring lanes read neighbouring records.
template <int DIM>
__global__ void __launch_bounds__(kBlock, 2) k_momentum_f32_split(DevBatch b, int fused) {
  chain_wait();
  constexpr int PARTS = 4;                             // 64 particles a block
  __shared__ SimDev s;
  __shared__ float sums[kBlock / 32][8][4][9 + 1];     // [warp][particle][chunk][sum]
  int cur = -1;
  const Particles& P = b.P;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane >> 3, g = lane & 7;
  for (int w = blockIdx.x; w < b.ntiles * PARTS; w += gridDim.x) {
    const Tile tl = b.tiles[w / PARTS];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    const int at = (w % PARTS) * (kBlock / 4) + warp * 8 + g;
    const int p = tl.start + at;
    const bool active = at < tl.count && p < s.p_off + dyn->nag && !dyn->frozen;
    int cnt = 0;
    MomentumPairs<DIM, false> m(s, P.RP);
    if (active) {
      m.load(P.XF[p], P.V[p], P.RP[p]);
      cnt = b.ncount[p];
    }
    Kahan k0, k1, k2;
    k0.zero();
    k1.zero();
    k2.zero();
    const int nch = (cnt + 3) >> 2;
    const int rounds = (int)(__reduce_max_sync(FULL, (unsigned)nch) + 3) >> 2;
    const int4* lbase = reinterpret_cast<const int4*>(b.nlist) + list_base4(p, b.list_cap4);
    int4 nxt = j < nch ? __ldg(lbase + (size_t)j * 32) : make_int4(0, 0, 0, 0);
    for (int r = 0; r < rounds; ++r) {
      const int c = 4 * r + j;
      const int4 ch = nxt;
      if (c + 4 < nch) nxt = __ldg(lbase + (size_t)(c + 4) * 32);
      if (c < nch) {
        m.template chunk<true>(P, ch, cnt - 4 * c);
        float* o = sums[warp][g][j];
        o[0] = m.cp0; o[1] = m.cp1; o[2] = m.cp2;
        o[3] = m.cd0; o[4] = m.cd1; o[5] = m.cd2;
        o[6] = m.cv0; o[7] = m.cv1; o[8] = m.cv2;
        m.clear();
      }
      __syncwarp();
      const int n = j < 3 ? min(nch - 4 * r, 4) : 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (q >= n) break;
        const float* o = sums[warp][g][q] + 3 * j;
        k0.add(o[0]);
        k1.add(o[1]);
        k2.add(o[2]);
      }
      __syncwarp();
    }
    double ms[9] = {k0.val(), k1.val(), k2.val()};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      ms[3 + d] = __shfl_down_sync(FULL, ms[d], 8);
      ms[6 + d] = __shfl_down_sync(FULL, ms[d], 16);
    }
    const bool close_here = fused && active && j == 0 && P.bdt_count[p] == 0;
    double dtc = 1.0e300;
    if (close_here) {
      double tpres[3] = {0, 0, 0};
      const double zero[3] = {0, 0, 0};
      const double4 v4 = P.V[p];
      const double2 rp = P.RP[p];
      const double vi[3] = {v4.x, v4.y, v4.z};
      momentum_f32_close<DIM, true>(s, b, dyn, p, ms, tpres, zero, zero, vi, rp.x, rp.y, 0, 0, dtc);
    }
    if (fused) {
      const double least = warp_min(dtc);
      if (lane == 0 && least < 1.0e300)
        atomicMin(&dyn->dtmin_bits, (unsigned long long)__double_as_longlong(least));
    }
    if (active && j == 0 && !close_here)
      for (int k = 0; k < 9; ++k) P.MSUM[(size_t)k * P.total_slots + p] = ms[k];
  }
}

// The finishing of particle p: its wall terms and closing.
// C1: as the FP64 form (k_momentum<3, F, true>): the first step completes
// and inverts B_ren_gradp in the wall pass; the renormalised pressure-
// gradient accumulator joins the ALE1 accumulator and the wall terms.
template <int DIM, bool FUSED, bool C1>
__device__ __forceinline__ void momentum_f32_finish(const SimDev& s, const DevBatch& b, SimDyn* dyn, int p,
                                                    double& dtc) {
  const Particles& P = b.P;
  double ms[9];
  for (int c = 0; c < 9; ++c) ms[c] = P.MSUM[(size_t)c * P.total_slots + p];
  double4 v4 = P.V[p];
  double2 rp = P.RP[p];
  const double vi[3] = {v4.x, v4.y, v4.z};
  const double rhoi = rp.x, pi = rp.y;
  const int nb = P.bdt_count[p];
  const int bstart = nb > 0 ? P.bdt_start[p] : 0;
  double tpres[3] = {0, 0, 0}, tdiss[3] = {0, 0, 0}, tvisc[3] = {0, 0, 0};
  const double* geff = dyn->geff;
  const bool c1 = C1 && DIM == 3 && s.c1_be;
  if (c1) {
    double B[9];
    const bool first = dyn->step == 0;
    load_b(P.BG, P.total_slots, p, B);
    if (nb > 0)
      me_boundary3d<true>(s, b, nb, bstart, vi, rhoi, pi, P.L[p], geff, tpres, tdiss, tvisc, B, first);
    else if (first)
      b_inversion(B, s.invb_det_thresh);
    if (first) store_b(P.BG, P.total_slots, p, B);
    // inter_EqMoto.f90:255-260: the pressure-gradient sum renormalised,
    // the ALE1 sum (the symmetric sum less it) as it is
    double g[3];
    for (int d = 0; d < 3; ++d) g[d] = P.MSUM[(size_t)(9 + d) * P.total_slots + p];
    const double al[3] = {ms[0] - g[0], ms[1] - g[1], ms[2] - g[2]};
    b_renormalise(B, g);
    for (int d = 0; d < 3; ++d) ms[d] = g[d] + al[d];
  } else if (nb > 0) {
    const int lam = P.L[p];
    if (DIM == 3) me_boundary3d(s, b, nb, bstart, vi, rhoi, pi, lam, geff, tpres, tdiss, tvisc);
    else me_boundary2d(s, b, nb, bstart, vi, rhoi, pi, lam, geff, tpres, tdiss, tvisc);
  }
  momentum_f32_close<DIM, FUSED>(s, b, dyn, p, ms, tpres, tdiss, tvisc, vi, rhoi, pi, nb, bstart, dtc);
}

template <int DIM, bool FUSED, bool C1 = false>
__global__ void __launch_bounds__(kBlock) k_momentum_f32_finish(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag;
    if (FUSED && active && dyn->frozen) {
      carry_record(P, p);
      active = false;
    }
    double dtc = 1.0e300;
    // in the fused step the pair launch has closed the particles without
    // close faces already (k_momentum_f32)
    if (FUSED && !C1 && active && P.bdt_count[p] == 0) active = false;
    if (active) momentum_f32_finish<DIM, FUSED, C1>(s, b, dyn, p, dtc);
    if (FUSED) {
      double m = warp_min(dtc);
      if ((threadIdx.x & 31) == 0 && m < 1.0e300)
        atomicMin(&dyn->dtmin_bits, (unsigned long long)__double_as_longlong(m));
    }
  }
}

// A particle's FP32c continuity pairs: its own values and the sum of the
// list chunk at hand.
template <int DIM>
struct ContinuityPairs {
  const SimDev& s;
  F32Const fc;
  RunCursor<DIM> rc;
  float4 xfi;
  float ckf, dz, vix, viy, viz, rhof, part;
  __device__ __forceinline__ ContinuityPairs(const SimDev& sim) : s(sim) {
    fc.load(sim);
    xfi = make_float4(0.f, 0.f, 0.f, 0.f);
    vix = viy = viz = ckf = part = 0.f;
    rhof = 1.f;
    dz = sim.dcdf[2];
  }
  __device__ __forceinline__ void load(const float4& x, const double4& v, double rho) {
    xfi = x;
    ckf = x.w;
    vix = (float)v.x;
    viy = (float)v.y;
    viz = (float)v.z;
    rhof = (float)rho;
  }
  __device__ __forceinline__ void pair(int e, const float4& xj, const float4& vj) {
    float d0, d1, d2;
    separation_f32<DIM>(s, rc, e, xj, xfi, ckf, dz, d0, d1, d2);
    float rr = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
    const float PK1 = kernel_pk1_f32(fc, rr);
    float c = rhof * vj.w * PK1;
    part = fmaf(c, fmaf(vj.z - viz, d2, fmaf(vj.y - viy, d1, (vj.x - vix) * d0)), part);
  }
  // pair for entries ea, eb on paired instructions (each half rounds
  // as the scalar instruction; x - y as fma(y, -1, x)), ea's term
  // accumulated before eb's
  __device__ __forceinline__ void pair2(int ea, int eb, const float4& xa, const float4& va, const float4& xb,
                                        const float4& vb) {
    const float2 m1 = make_float2(-1.f, -1.f);
    rc.update(s, (int)((unsigned)ea >> kSlotBits));
    const float dxa = rc.Dx, dya = rc.Dy;
    rc.update(s, (int)((unsigned)eb >> kSlotBits));
    const float2 Dx = make_float2(dxa, rc.Dx), Dy = make_float2(dya, rc.Dy);
    const float2 d0 = __fadd2_rn(Dx, __ffma2_rn(make_float2(xa.x, xb.x), m1, make_float2(xfi.x, xfi.x)));
    const float2 d1 = (DIM == 3)
                          ? __fadd2_rn(Dy, __ffma2_rn(make_float2(xa.y, xb.y), m1, make_float2(xfi.y, xfi.y)))
                          : make_float2(0.f, 0.f);
    const float2 dk = __ffma2_rn(make_float2(xa.w, xb.w), m1, make_float2(ckf, ckf));
    const float2 d2 = __fadd2_rn(__fmul2_rn(dk, make_float2(dz, dz)),
                                 __ffma2_rn(make_float2(xa.z, xb.z), m1, make_float2(xfi.z, xfi.z)));
    const float2 rr = __ffma2_rn(d2, d2, __ffma2_rn(d1, d1, __fmul2_rn(d0, d0)));
    // kernel_pk1_f32
    const float2 rq = make_float2(fmaxf(rr.x, 1.0e-30f), fmaxf(rr.y, 1.0e-30f));
    const float2 r = __fmul2_rn(rq, make_float2(rsqrt_approx(rq.x), rsqrt_approx(rq.y)));
    const float2 q = __fmul2_rn(r, make_float2(fc.hinv, fc.hinv));
    const float2 q2 = __fmul2_rn(rr, make_float2(fc.h2inv, fc.h2inv));
    const float2 glo = __ffma2_rn(make_float2(1.5f, 1.5f), q2, __fmul2_rn(make_float2(-2.0f, -2.0f), q));
    const float2 ghi = __ffma2_rn(make_float2(-0.5f, -0.5f), q2,
                                  __ffma2_rn(make_float2(2.0f, 2.0f), q, make_float2(-2.0f, -2.0f)));
    const float2 g = make_float2(q.x < 1.0f ? glo.x : ghi.x, q.y < 1.0f ? glo.y : ghi.y);
    const float2 ra = __fadd2_rn(r, make_float2(fc.eta, fc.eta));
    const float2 PK1 = __fmul2_rn(__fmul2_rn(g, make_float2(fc.ke, fc.ke)),
                                  make_float2(rcp_approx(ra.x), rcp_approx(ra.y)));
    const float2 c = __fmul2_rn(__fmul2_rn(make_float2(rhof, rhof), make_float2(va.w, vb.w)), PK1);
    const float2 dv0 = __ffma2_rn(make_float2(vix, vix), m1, make_float2(va.x, vb.x));
    const float2 dv1 = __ffma2_rn(make_float2(viy, viy), m1, make_float2(va.y, vb.y));
    const float2 dv2 = __ffma2_rn(make_float2(viz, viz), m1, make_float2(va.z, vb.z));
    const float2 u = __ffma2_rn(dv2, d2, __ffma2_rn(dv1, d1, __fmul2_rn(dv0, d0)));
    part = fmaf(c.x, u.x, part);
    part = fmaf(c.y, u.y, part);
  }
  // the entries of a chunk, rem of them, their records requested together
  template <bool PAIRED>
  __device__ __forceinline__ void chunk(const Particles& P, const int4& ch, int rem) {
    const int q0 = ch.x & kSlotMask, q1 = ch.y & kSlotMask, q2 = ch.z & kSlotMask, q3 = ch.w & kSlotMask;
    float4 x0, v0, x1, v1, x2, v2, x3, v3;
    x0 = __ldg(P.XF + q0); v0 = __ldg(P.VF + q0);
    if (rem > 1) { x1 = __ldg(P.XF + q1); v1 = __ldg(P.VF + q1); }
    if (rem > 2) { x2 = __ldg(P.XF + q2); v2 = __ldg(P.VF + q2); }
    if (rem > 3) { x3 = __ldg(P.XF + q3); v3 = __ldg(P.VF + q3); }
    if (PAIRED) {
      if (rem > 1) pair2(ch.x, ch.y, x0, v0, x1, v1);
      else pair(ch.x, x0, v0);
      if (rem > 3) pair2(ch.z, ch.w, x2, v2, x3, v3);
      else if (rem > 2) pair(ch.z, x2, v2);
    } else {
      pair(ch.x, x0, v0);
      if (rem > 1) pair(ch.y, x1, v1);
      if (rem > 2) pair(ch.z, x2, v2);
      if (rem > 3) pair(ch.w, x3, v3);
    }
  }
};

// Continuity, FP32c form, in two launches so that the pair sum need not
// wait for the boundary data: k_continuity_f32 writes the compensated pair
// sum of each particle to DDEN, and k_continuity_f32_finish, once the
// boundary data exist, forms dden = (SA-SPH wall term) - (pair sum) and, in
// the fused step, Leapfrog_continuity and the EoS.
// DIVU (C1_BE and C1_divu, 3D): a simulation that renormalises sums the
// whole velocity-gradient tensor, G(a, k) = sum rho_i (m_j / rho_j) PK1
// (v_j - v_i)_a r_k, nine compensated sums written to MSUM, which the
// finishing launch renormalises with B_ren_divu (Continuity_Equation.f90:
// 119-126,201-217); the others of the batch sum as without it.
// BATCH (not with DIVU): a list chunk's eight neighbour records requested
// before the chunk's arithmetic, at 3 blocks per SM; the same sums.
// PAIRED (with BATCH): two entries' terms on paired FP32 instructions
// (pair2), the same bits as two calls of `pair`.
template <int DIM, bool DIVU = false, bool BATCH = false, bool PAIRED = false>
__global__ void __launch_bounds__(kBlock, DIVU ? 2 : (BATCH ? 3 : 5)) k_continuity_f32(DevBatch b) {
  chain_wait();
  static_assert(!PAIRED || (BATCH && !DIVU), "the paired loop is a batched, non-C1 shape");
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen;
    int cnt = 0;
    ContinuityPairs<DIM> m(s);
    if (active) {
      m.load(P.XF[p], P.V[p], P.RP[p].x);
      cnt = b.ncount[p];
    }
    const bool tensor = DIVU && DIM == 3 && s.c1_be && s.c1_divu;
    Kahan sum;
    sum.zero();
    Kahan gs[9];
    float gp[9];
#pragma unroll
    for (int a = 0; a < 9; ++a) {
      gs[a].zero();
      gp[a] = 0.f;
    }
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    if (BATCH && !DIVU) {
      const int nch = (cnt + 3) >> 2, nchmax = (nmax + 3) >> 2;
      const int4* lbase = reinterpret_cast<const int4*>(b.nlist) + list_base4(p, b.list_cap4);
      int4 nxt = nch > 0 ? __ldg(lbase) : make_int4(0, 0, 0, 0);
      for (int c = 0; c < nchmax; ++c) {
        const int4 ch = nxt;
        if (c + 1 < nch) nxt = __ldg(lbase + (size_t)(c + 1) * 32);
        if (c >= nch) continue;
        const int rem = cnt - 4 * c;
        m.template chunk<PAIRED>(P, ch, rem);
        sum.add(m.part);   // 4-entry partial sums, compensated into sum
        m.part = 0.f;
      }
    }
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, (BATCH && !DIVU) ? 0 : cnt);
    for (int k = 0; k < ((BATCH && !DIVU) ? 0 : nmax); ++k) {
      const int e = lr.get(k);
      if (k >= cnt) continue;
      const float4 xj = __ldg(P.XF + (e & kSlotMask)), vj = __ldg(P.VF + (e & kSlotMask));
      float d0, d1, d2;
      separation_f32<DIM>(s, m.rc, e, xj, m.xfi, m.ckf, m.dz, d0, d1, d2);
      float rr = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
      const float PK1 = kernel_pk1_f32(m.fc, rr);
      float c = m.rhof * vj.w * PK1;    // rho_i (m_j / rho_j) PK1
      const bool flush = (k & 3) == 3 || k == cnt - 1;
      if (DIVU && tensor) {
        const float cv[3] = {c * (vj.x - m.vix), c * (vj.y - m.viy), c * (vj.z - m.viz)};
        const float dd[3] = {d0, d1, d2};
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
          for (int q = 0; q < 3; ++q) gp[3 * a + q] = fmaf(cv[a], dd[q], gp[3 * a + q]);
        if (flush) {
#pragma unroll
          for (int a = 0; a < 9; ++a) {
            gs[a].add(gp[a]);
            gp[a] = 0.f;
          }
        }
      } else {
        m.part = fmaf(c, fmaf(vj.z - m.viz, d2, fmaf(vj.y - m.viy, d1, (vj.x - m.vix) * d0)), m.part);
        if (flush) {
          sum.add(m.part);
          m.part = 0.f;
        }
      }
    }
    if (active) {
      if (DIVU && tensor) {
#pragma unroll
        for (int a = 0; a < 9; ++a) P.MSUM[(size_t)a * P.total_slots + p] = gs[a].val();
      } else {
        P.DDEN[p] = sum.val();
      }
    }
  }
}

// k_continuity_f32 with four lanes to a particle (k_momentum_f32_split's
// scheme); the chunk sums go round by shuffles.
template <int DIM>
__global__ void __launch_bounds__(kBlock, 3) k_continuity_f32_split(DevBatch b) {
  chain_wait();
  constexpr int PARTS = 4;
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, j = lane >> 3, g = lane & 7;
  for (int w = blockIdx.x; w < b.ntiles * PARTS; w += gridDim.x) {
    const Tile tl = b.tiles[w / PARTS];
    load_sim(s, b.sims, tl.sim, cur);
    const SimDyn* dyn = b.dyn + tl.sim;
    const int at = (w % PARTS) * (kBlock / 4) + warp * 8 + g;
    const int p = tl.start + at;
    const bool active = at < tl.count && p < s.p_off + dyn->nag && !dyn->frozen;
    int cnt = 0;
    ContinuityPairs<DIM> m(s);
    if (active) {
      m.load(P.XF[p], P.V[p], P.RP[p].x);
      cnt = b.ncount[p];
    }
    Kahan sum;
    sum.zero();
    const int nch = (cnt + 3) >> 2;
    const int rounds = (int)(__reduce_max_sync(FULL, (unsigned)nch) + 3) >> 2;
    const int4* lbase = reinterpret_cast<const int4*>(b.nlist) + list_base4(p, b.list_cap4);
    int4 nxt = j < nch ? __ldg(lbase + (size_t)j * 32) : make_int4(0, 0, 0, 0);
    for (int r = 0; r < rounds; ++r) {
      const int c = 4 * r + j;
      const int4 ch = nxt;
      if (c + 4 < nch) nxt = __ldg(lbase + (size_t)(c + 4) * 32);
      m.part = 0.f;
      if (c < nch) m.template chunk<true>(P, ch, cnt - 4 * c);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float v = __shfl_sync(FULL, m.part, 8 * q + g);
        if (4 * r + q < nch) sum.add(v);
      }
    }
    if (active && j == 0) P.DDEN[p] = sum.val();
  }
}

// C1 (3D): the frontiers complete both matrices, which are inverted for
// every particle (continuity_boundary_c1, FP64); with C1_divu the pair
// tensor is renormalised with B_ren_divu and its trace enters drho/dt.
template <int DIM, bool FUSED, bool C1 = false>
__global__ void __launch_bounds__(kBlock) k_continuity_f32_finish(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    if (!(threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen)) continue;
    const double rhoi = P.RP[p].x;
    double dden = 0.0;
    const int nb = P.bdt_count[p];
    // read by the wall terms alone; with C1 loaded always: a selected load takes
    // the launch from 127 registers to 154, from two blocks an SM to one
    double4 vi = make_double4(0.0, 0.0, 0.0, 0.0);
    if (C1 || nb > 0) vi = P.V[p];
    if (C1 && DIM == 3 && s.c1_be) {
      dden = continuity_boundary_c1(s, b, dyn, nb, nb > 0 ? P.bdt_start[p] : 0, vi, rhoi, p);
      if (s.c1_divu) {
        double B[9], g[3][3];
        load_b(P.BD, P.total_slots, p, B);
        for (int a = 0; a < 3; ++a) {
          for (int q = 0; q < 3; ++q) g[a][q] = P.MSUM[(size_t)(3 * a + q) * P.total_slots + p];
          b_renormalise(B, g[a]);
        }
        dden = dden - (g[0][0] + g[1][1] + g[2][2]);
      } else {
        dden = dden - P.DDEN[p];
      }
    } else {
      if (nb > 0) dden = continuity_boundary<DIM>(s, b, dyn, nb, P.bdt_start[p], vi, rhoi);
      dden = dden - P.DDEN[p];
    }
    if (FUSED) {
      double rho = rhoi + dyn->dt * dden;
      if (s.density_thresholds == 1) {
        if (rho < 0.9 * s.den0) rho = 0.9 * s.den0;
        if (rho > 1.1 * s.den0) rho = 1.1 * s.den0;
      }
      double pr = s.k_over_rho0 * (rho - s.den0) + s.p_ref;
      P.RP[p] = make_double2(rho, pr);
      const double m = P.X[p].w;
      if (b.smooths) P.RF[p] = make_float4((float)rho, (float)(pr / (rho * rho)), (float)m, 0.f);
      // the next momentum pass's records: the new density, and m/rho in
      // VF.w (the pair sums of this pass, which read the old one, are done)
      P.RM[p] = make_float2((float)rho, (float)(pr / (rho * rho)));
      P.VF[p].w = (float)(m / rho);
    } else {
      P.DDEN[p] = dden;
    }
  }
}

// FP32 copies of velocity, density and pressure after an in-place update
// of the FP64 state by the per-call ABI.
__global__ void k_refresh_f32(DevBatch b) {
  __shared__ SimDev s;
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    double4 x = b.P.X[p];
    double4 v = b.P.V[p];
    double2 rp = b.P.RP[p];
    // m/rho of the current density (after a pressure smoothing V.w still
    // holds the sort's; where they agree this is the same division)
    b.P.VF[p] = make_float4((float)v.x, (float)v.y, (float)v.z, (float)(x.w / rp.x));
    b.P.RF[p] = make_float4((float)rp.x, (float)(rp.y / (rp.x * rp.x)), (float)x.w, 0.f);
    b.P.RM[p] = make_float2((float)rp.x, (float)(rp.y / (rp.x * rp.x)));
  }
}

// ==========================================================================
// Partial smoothing (input_any_t%TetaV, %TetaP > 0), FP64 in both forms.
// The reference's neighbour list includes the particle itself; the lists
// here leave it out, so its term is added where the reference's order puts
// it: before the first entry past (centre run, own slot).
// ==========================================================================

// PartKernel(4) of CalcVarLength.f90:241-268: the kernel value W = wu coefke.
// NaN for a NaN separation: the smoothing sums multiply W by values that need
// not be NaN themselves, and the pair is not to be passed over.
__device__ __forceinline__ double kernel_w(const SimDev& s, double rr) {
  double r = sqrt(rr);
  double q = div_rn_unsigned0(r, s.h, s.rcp_h);
  double q2 = div_rn_unsigned0(rr, s.squareh, s.rcp_squareh);
  if (at_least_two(q) && !isnan(q)) return 0.0;
  double wu = 0.666666667 + q2 * (q * 0.5 - 1.0);
  if (at_least_one(q)) wu = (2.0 - q) * (2.0 - q) * (2.0 - q) * 0.166666666667;
  return wu * s.coefke;
}

// velocity_smoothing_SA_SPH_3D.f90:61-125 / _2D.f90:66-117 (fixe/tapi
// walls, slip mode 1): adds the wall terms of particle p to var.
template <int DIM>
__device__ __forceinline__ void smoothing_wall_velocity(const SimDev& s, const DevBatch& b, int p, const double4& vi,
                                                        double* var) {
  const Particles& P = b.P;
  const int nb = P.bdt_count[p];
  const int bstart = nb > 0 ? P.bdt_start[p] : 0;
  for (int u = 0; u < nb; ++u) {
    const BdtEntry& e = P.bdt[bstart + u];
    if (DIM == 3) {
      const FaceDev& f = b.faces[s.face_off + e.clobonum - 1];
      const double vv[3] = {vi.x, vi.y, vi.z};
      double DVGlo[3], DVLoc[3], BCLoc[3];
      for (int i = 0; i < 3; ++i) DVGlo[i] = 2.0 * (f.velocity[i] - vv[i]);
      for (int i = 0; i < 3; ++i) {
        double a = 0.0;
        for (int j = 0; j < 3; ++j) a = a + f.T[j][i] * DVGlo[j];
        DVLoc[i] = a;
      }
      double IntWdV = e.bi[1];
      BCLoc[0] = DVLoc[0] * IntWdV * f.slip;
      BCLoc[1] = DVLoc[1] * IntWdV * f.slip;
      BCLoc[2] = DVLoc[2] * IntWdV;
      for (int i = 0; i < 3; ++i) {
        double g = 0.0;
        for (int j = 0; j < 3; ++j) g = g + f.T[i][j] * BCLoc[j];
        var[i] = var[i] + g;
      }
    } else {
      const SideDev& S = b.sides[s.side_off + e.clobonum - 1];
      double DVGlo0 = 2.0 * (S.velocity[0] - vi.x), DVGlo1 = 2.0 * (S.velocity[2] - vi.z);
      double DVLoc0 = S.sss[0] * DVGlo0 + S.sss[1] * DVGlo1;
      double DVLoc1 = S.nnn[0] * DVGlo0 + S.nnn[1] * DVGlo1;
      double IntWdV = e.bi[2];
      double BCLoc0 = DVLoc0 * IntWdV * S.slip;
      double BCLoc1 = DVLoc1 * IntWdV;
      var[0] = var[0] + (S.sss[0] * BCLoc0 + S.nnn[0] * BCLoc1);
      var[2] = var[2] + (S.sss[1] * BCLoc0 + S.nnn[1] * BCLoc1);
    }
  }
}

// The wall terms and the update of PressureSmoothing_3D.f90:111-134 /
// _2D.f90:140-212 for particle p with pair sums sompW and AppUnity: the
// smoothed pressure.
template <int DIM>
__device__ __forceinline__ double smoothing_pressure(const SimDev& s, const DevBatch& b, const SimDyn* dyn, int p,
                                                     double pi, double sompW, double AppUnity) {
  const Particles& P = b.P;
  const double TetaP1 = s.teta_p * s.celerita * dyn->dt / s.h;
  const double p0i = s.p_ref;
  const int nb = P.bdt_count[p];
  const int bstart = nb > 0 ? P.bdt_start[p] : 0;
  double vpres;
  if (DIM == 3) {
    for (int u = 0; u < nb; ++u) {
      const BdtEntry& e = P.bdt[bstart + u];
      if (e.loc[2] > 0.0) AppUnity = AppUnity + e.bi[1];
    }
    double DiffP = (AppUnity < 0.95) ? sompW + (p0i - pi) * (1.0 - AppUnity) : sompW / AppUnity;
    vpres = pi + TetaP1 * DiffP;
  } else {
    const double* g = dyn->geff;
    double VIntWdV_FT = 0.0;
    for (int u = 0; u < nb; ++u) {
      const BdtEntry& e = P.bdt[bstart + u];
      const SideDev& S = b.sides[s.side_off + e.clobonum - 1];
      double mf0 = S.sss[0] * g[0] + S.sss[1] * g[2];
      double mf1 = S.nnn[0] * g[0] + S.nnn[1] * g[2];
      VIntWdV_FT = VIntWdV_FT + e.bi[1];
      sompW = sompW + s.den0 * (mf0 * e.bi[3] + mf1 * e.bi[4]);
    }
    AppUnity = AppUnity + VIntWdV_FT + 0.0 + 0.0 + 0.0;
    vpres = pi + TetaP1 * (sompW + (pi - pi) * 0.0 + (pi - pi) * 0.0 + (p0i - pi) * (1.0 - AppUnity));
  }
  return vpres;
}

// velocity_smoothing.f90:85-132 with velocity_smoothing_SA_SPH_3D.f90:61-125
// / _2D.f90:66-117 (fixe/tapi walls, slip mode 1): ACC = var, the smoothing
// increment, from the velocities `vel` (the step's leapfrog velocities).
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_velocity_smoothing(DevBatch b, const double4* __restrict__ vel) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  constexpr int RC = (DIM == 3) ? 4 : 1;   // the particle's own column run
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    const bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen && s.teta_v > 1.0e-9;
    const int cnt = active ? b.ncount[p] : 0;
    double var[3] = {0.0, 0.0, 0.0};
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0), vi = xi;
    double self_w = 0.0;
    if (active) {
      xi = P.X[p];
      vi = vel[p];
      self_w = xi.w * kernel_w(s, 0.0) / P.RP[p].x;
    }
    bool self_done = !active;
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    for (int k = 0; k < nmax; ++k) {
      int e = lr.get(k);
      if (k >= cnt) continue;
      int q = e & kSlotMask;
      int r = (int)((unsigned)e >> kSlotBits);
      if (!self_done && (r > RC || (r == RC && q > p))) {
        var[0] = var[0] + (vi.x - vi.x) * self_w;
        var[1] = var[1] + (vi.y - vi.y) * self_w;
        var[2] = var[2] + (vi.z - vi.z) * self_w;
        self_done = true;
      }
      double4 xj = P.X[q];
      double r0 = xi.x - xj.x, r1 = xi.y - xj.y, r2 = xi.z - xj.z;
      double rr = r0 * r0 + r1 * r1 + r2 * r2;
      double pesoj = xj.w * kernel_w(s, rr) / P.RP[q].x;
      double4 vj = vel[q];
      var[0] = var[0] + (vj.x - vi.x) * pesoj;
      var[1] = var[1] + (vj.y - vi.y) * pesoj;
      var[2] = var[2] + (vj.z - vi.z) * pesoj;
    }
    if (!active) continue;
    if (!self_done) {
      var[0] = var[0] + (vi.x - vi.x) * self_w;
      var[1] = var[1] + (vi.y - vi.y) * self_w;
      var[2] = var[2] + (vi.z - vi.z) * self_w;
    }
    smoothing_wall_velocity<DIM>(s, b, p, vi, var);
    P.ACC[p] = make_double4(var[0], var[1], var[2], 0.0);
  }
}

// The FP32c form's smoothing sums: the same terms in FP32 from the FP32
// records (XF, RF, and VF2, the leapfrog velocities the momentum pass
// writes in FP32) with compensated 4-entry chunk sums, the pressure
// differences formed in FP64 first; the particle's own term (zero for
// velocities) and the wall terms in FP64.
__device__ __forceinline__ float kernel_w_f32(float rr, float hinv, float coefke) {
  float r = rr * rsqrtf(rr);
  float q = r * hinv;
  if (!(q < 2.0f)) return 0.f;
  float wu = (q < 1.0f) ? fmaf(q * q, fmaf(q, 0.5f, -1.0f), 0.666666667f)
                        : (2.0f - q) * (2.0f - q) * (2.0f - q) * (1.0f / 6.0f);
  return wu * coefke;
}

template <int DIM>
__global__ void __launch_bounds__(kBlock, 4) k_velocity_smoothing_f32(DevBatch b, const double4* __restrict__ vel) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    const bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen && s.teta_v > 1.0e-9;
    const float hinv = (float)(1.0 / s.h), coefke = (float)s.coefke;
    int cnt = 0;
    float4 xfi = make_float4(0.f, 0.f, 0.f, 0.f);
    double4 vi = make_double4(0.0, 0.0, 0.0, 0.0);
    if (active) {
      xfi = P.XF[p];
      vi = vel[p];
      cnt = b.ncount[p];
    }
    const float ckf = xfi.w, dz = s.dcdf[2];
    RunCursor<DIM> rc;
    const float4 vif = make_float4((float)vi.x, (float)vi.y, (float)vi.z, 0.f);
    Kahan k0, k1, k2;
    k0.zero(); k1.zero(); k2.zero();
    float c0 = 0.f, c1 = 0.f, c2 = 0.f;
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    for (int k = 0; k < nmax; ++k) {
      int e = lr.get(k);
      if (k >= cnt) continue;
      int q = e & kSlotMask;
      const float4 xj = P.XF[q], rfj = P.RF[q], vj = P.VF2[q];
      float d0, d1, d2;
      separation_f32<DIM>(s, rc, e, xj, xfi, ckf, dz, d0, d1, d2);
      float rr = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
      float pes = __fdividef(rfj.z * kernel_w_f32(rr, hinv, coefke), rfj.x);
      c0 = fmaf(vj.x - vif.x, pes, c0);
      if (DIM == 3) c1 = fmaf(vj.y - vif.y, pes, c1);
      c2 = fmaf(vj.z - vif.z, pes, c2);
      if ((k & 3) == 3 || k == cnt - 1) {
        k0.add(c0); k1.add(c1); k2.add(c2);
        c0 = c1 = c2 = 0.f;
      }
    }
    if (!active) continue;
    double var[3] = {k0.val(), k1.val(), k2.val()};
    smoothing_wall_velocity<DIM>(s, b, p, vi, var);
    P.ACC[p] = make_double4(var[0], var[1], var[2], 0.0);
  }
}

template <int DIM>
__global__ void __launch_bounds__(kBlock, 4) k_pressure_smoothing_f32(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    const bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen && s.teta_p > 0.0;
    const float hinv = (float)(1.0 / s.h), coefke = (float)s.coefke;
    int cnt = 0;
    float4 xfi = make_float4(0.f, 0.f, 0.f, 0.f);
    double pi = 0.0;
    float self = 0.f;
    if (active) {
      xfi = P.XF[p];
      const float4 rfi = P.RF[p];
      pi = P.RP[p].y;
      self = __fdividef(rfi.z * (0.666666667f * coefke), rfi.x);
      cnt = b.ncount[p];
    }
    const float ckf = xfi.w, dz = s.dcdf[2];
    RunCursor<DIM> rc;
    Kahan ka, ks;
    ka.zero();
    ks.zero();
    float ca = self, cs = 0.f;
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    for (int k = 0; k < nmax; ++k) {
      int e = lr.get(k);
      if (k >= cnt) continue;
      int q = e & kSlotMask;
      const float4 xj = P.XF[q], rfj = P.RF[q];
      const float dp = (float)(P.RP[q].y - pi);
      float d0, d1, d2;
      separation_f32<DIM>(s, rc, e, xj, xfi, ckf, dz, d0, d1, d2);
      float rr = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
      float pes = __fdividef(rfj.z * kernel_w_f32(rr, hinv, coefke), rfj.x);
      ca += pes;
      cs = fmaf(dp, pes, cs);
      if ((k & 3) == 3 || k == cnt - 1) {
        ka.add(ca);
        ks.add(cs);
        ca = cs = 0.f;
      }
    }
    if (!active) continue;
    if (cnt == 0) ka.add(ca);   // the particle's own term alone
    P.DDEN[p] = smoothing_pressure<DIM>(s, b, dyn, p, pi, ks.val(), ka.val());
  }
}

// velocity_smoothing_2.f90:87-101 with TetaV > 1e-9: vel = vel + TetaV1 var.
// FUSED (the step graph): on the momentum pass's record V2, then
// Leapfrog_trajectories into X2 and the CFL minimum of the smoothed
// velocities; otherwise in place on V (the per-call ABI).
template <bool FUSED>
__global__ void __launch_bounds__(kBlock) k_velocity_smoothing_apply(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    const bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen && s.teta_v > 1.0e-9;
    double dtc = 1.0e300;
    if (active) {
      const double TetaV1 = s.teta_v * s.celerita * dyn->dt / s.h;
      const double4 var = P.ACC[p];
      double4 v = FUSED ? P.V2[p] : P.V[p];
      v.x = v.x + TetaV1 * var.x;
      v.y = v.y + TetaV1 * var.y;
      v.z = v.z + TetaV1 * var.z;
      if (FUSED) {
        P.V2[p] = v;
        const double4 x = P.X[p];
        const double dt = dyn->dt;
        P.X2[p] = make_double4(x.x + dt * v.x, x.y + dt * v.y, x.z + dt * v.z, x.w);
        double U = sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
        dtc = s.cfl * 2.0 * s.h / (s.celerita + U);
      } else {
        P.V[p] = v;
      }
    }
    if (FUSED) {
      double m = warp_min(dtc);
      if ((threadIdx.x & 31) == 0 && m < 1.0e300)
        atomicMin(&dyn->dtmin_bits, (unsigned long long)__double_as_longlong(m));
    }
  }
}

// PressureSmoothing_3D.f90:88-134 / PressureSmoothing_2D.f90:102-212
// (SmoothVersion "b", fixe/tapi walls): DDEN = the smoothed pressure, from
// the pressures and densities after the step's EoS.
template <int DIM>
__global__ void __launch_bounds__(kBlock) k_pressure_smoothing(DevBatch b) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  constexpr int RC = (DIM == 3) ? 4 : 1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    const bool active = threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen && s.teta_p > 0.0;
    const int cnt = active ? b.ncount[p] : 0;
    double4 xi = make_double4(0.0, 0.0, 0.0, 0.0);
    double pi = 0.0, self_w = 0.0, sompW = 0.0, AppUnity = 0.0;
    if (active) {
      xi = P.X[p];
      double2 rp = P.RP[p];
      pi = rp.y;
      self_w = xi.w * kernel_w(s, 0.0) / rp.x;
    }
    bool self_done = !active;
    ListPrefetcher lr;
    lr.init(b.nlist, p, b.list_cap4, cnt);
    const int nmax = __reduce_max_sync(0xffffffffu, (unsigned)cnt);
    prefetch_list_l2(b.nlist, p, b.list_cap4, nmax);
    for (int k = 0; k < nmax; ++k) {
      int e = lr.get(k);
      if (k >= cnt) continue;
      int q = e & kSlotMask;
      int r = (int)((unsigned)e >> kSlotBits);
      if (!self_done && (r > RC || (r == RC && q > p))) {
        AppUnity = AppUnity + self_w;
        sompW = sompW + (pi - pi) * self_w;
        self_done = true;
      }
      double4 xj = P.X[q];
      double r0 = xi.x - xj.x, r1 = xi.y - xj.y, r2 = xi.z - xj.z;
      double rr = r0 * r0 + r1 * r1 + r2 * r2;
      double2 rpj = P.RP[q];
      double pesoj = xj.w * kernel_w(s, rr) / rpj.x;
      AppUnity = AppUnity + pesoj;
      sompW = sompW + (rpj.y - pi) * pesoj;
    }
    if (!active) continue;
    if (!self_done) {
      AppUnity = AppUnity + self_w;
      sompW = sompW + (pi - pi) * self_w;
    }
    P.DDEN[p] = smoothing_pressure<DIM>(s, b, dyn, p, pi, sompW, AppUnity);
  }
}

// PressureSmoothing_3D.f90:137-158 / _2D.f90:216-233: p = the smoothed
// pressure, density from the inverse EoS (EoS_barotropic_linear.f90:54),
// and the FP32 record of the FP32c form.
__global__ void __launch_bounds__(kBlock) k_pressure_smoothing_apply(DevBatch b, int refresh_f32) {
  chain_wait();
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    SimDyn* dyn = b.dyn + tl.sim;
    int p = tl.start + threadIdx.x;
    if (!(threadIdx.x < tl.count && p < s.p_off + dyn->nag && !dyn->frozen && s.teta_p > 0.0)) continue;
    double pr = P.DDEN[p];
    double rho = s.den0 * (1.0 + (pr - s.p_ref) / s.eps);
    P.RP[p] = make_double2(rho, pr);
    if (refresh_f32) {
      const double m = P.X[p].w;
      P.RF[p] = make_float4((float)rho, (float)(pr / (rho * rho)), (float)m, 0.f);
      P.RM[p] = make_float2((float)rho, (float)(pr / (rho * rho)));
      P.VF[p].w = (float)(m / rho);
    }
  }
}

// ==========================================================================
// Fine-grained integration kernels (used by the per-call C ABI)
// ==========================================================================
__global__ void k_leapfrog_momentum(DevBatch b) {
  __shared__ SimDev s;
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    double dtvel = b.dyn[tl.sim].dtvel;
    double4 v = b.P.V[p];
    double4 a = b.P.ACC[p];
    v.x = v.x + dtvel * a.x;
    v.y = v.y + dtvel * a.y;
    v.z = v.z + dtvel * a.z;
    b.P.V[p] = v;
    if (b.P.VF2) b.P.VF2[p] = make_float4((float)v.x, (float)v.y, (float)v.z, 0.f);
  }
}

__global__ void k_leapfrog_trajectories(DevBatch b) {
  __shared__ SimDev s;
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    double dt = b.dyn[tl.sim].dt;
    double4 x = b.P.X[p];
    double4 v = b.P.V[p];
    x.x = x.x + dt * v.x;
    x.y = x.y + dt * v.y;
    x.z = x.z + dt * v.z;
    b.P.X[p] = x;   // the screening copies are rebuilt by the next sph_ord_grid
  }
}

__global__ void k_leapfrog_continuity(DevBatch b) {
  __shared__ SimDev s;
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    double2 rp = b.P.RP[p];
    double rho = rp.x + b.dyn[tl.sim].dt * b.P.DDEN[p];
    if (s.density_thresholds == 1) {
      if (rho < 0.9 * s.den0) rho = 0.9 * s.den0;
      if (rho > 1.1 * s.den0) rho = 1.1 * s.den0;
    }
    b.P.RP[p] = make_double2(rho, rp.y);
    double4 v = b.P.V[p];
    v.w = b.P.X[p].w / rho;
    b.P.V[p] = v;
  }
}

__global__ void k_eos(DevBatch b) {
  __shared__ SimDev s;
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    if (b.dyn[tl.sim].step < 0) continue;   // EoS_fluid_loop.f90:61 (on_going_time_step > 0)
    double2 rp = b.P.RP[p];
    rp.y = s.k_over_rho0 * (rp.x - s.den0) + s.p_ref;
    b.P.RP[p] = rp;
  }
}

// CFL minimum of time_step_duration.f90:86-110 over the current velocities.
__global__ void k_dt_reduce(DevBatch b) {
  __shared__ SimDev s;
  __shared__ double red[kBlock / 32];
  int cur = -1;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    double dtc = 1.0e300;
    if (threadIdx.x < tl.count && p < s.p_off + b.dyn[tl.sim].nag) {
      double4 v = b.P.V[p];
      double U = sqrt(v.x * v.x + v.y * v.y + v.z * v.z);
      dtc = s.cfl * 2.0 * s.h / (s.celerita + U);
    }
    double m = warp_min(dtc);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
      double mm = red[0];
      for (int w = 1; w < kBlock / 32; ++w) mm = fmin(mm, red[w]);
      if (mm < 1.0e300) atomicMin(&b.dyn[tl.sim].dtmin_bits, (unsigned long long)__double_as_longlong(mm));
    }
    __syncthreads();
  }
}

// time_step_duration.f90:74-123 closing formula for on_going_time_step.
__device__ void tsd_close(const SimDev& s, SimDyn& d, double dtmin_cfl, int on_going) {
  double dtmin = kMaxPositive;
  double dt_vis = kMaxPositive;
  double dt;
  if (d.nag == 0) {
    dt = 0.0;
  } else {
    if (s.kin_visc > 1.0e-24) {
      dt_vis = s.vsc_coeff * s.squareh / (0.5 * s.kin_visc);
      dtmin = fmin(dtmin, dt_vis);
    }
    dtmin = fmin(dtmin, fmin(dtmin_cfl, dt_vis));
    if (s.dt_alfa_mon) {
      double visc_mon = s.alfa_mon * s.celerita * s.h / s.den0;
      double dt_mon = s.squareh / (0.5 * visc_mon);
      dtmin = fmin(dtmin, fmin(kMaxPositive, dt_mon));
    }
    if (on_going == 0) dt = dtmin;
    else dt = (1.0 - s.pesodt) * dtmin + s.pesodt * d.dt_average;
  }
  if (on_going == 0) d.dt_average = dt;
  else d.dt_average = (d.dt_average * (on_going - 1) + dt) / on_going;
  d.dt = dt;
}

// mode 0: IC.  time_step_loop.f90:173 evaluates dt with on_going_time_step
//         = -999, then the first iteration (time_step_loop.f90:182-185)
//         evaluates it again for step 1 from the same velocities.
// mode 1: end of a step: advance the simulation time and evaluate the dt of
//         the next iteration (its time_step_duration sees the velocities
//         this step left).
// Between steps the state keeps: step = completed steps, time = sum of their
// dt, dt = dt of the next step, dt_prev = dt of the last step.
// Sine of the tank forcing phase, written out so that host and device give
// the same bits: x is reduced by the nearest multiple of 2 pi into
// [-pi, pi], folded into [-pi/2, pi/2] by sin(r) = sin(+-pi - r), and the
// Taylor series of sin is summed to the r^23 term in nested form,
// r (1 - r^2/(2*3) (1 - r^2/(4*5) (...))), truncation below 1e-20 there.
// Every operation is a correctly rounded IEEE operation.
__device__ __forceinline__ double forcing_sin(double x) {
  const double two_pi = 6.283185307179586, pi = 3.141592653589793, half_pi = 1.5707963267948966;
  double k = rint(x / two_pi);
  double r = x - k * two_pi;
  if (r > half_pi) r = pi - r;
  else if (r < -half_pi) r = -pi - r;
  double r2 = r * r;
  double t = 1.0;
  for (int n = 22; n >= 2; n -= 2) t = 1.0 - r2 / (double)(n * (n + 1)) * t;
  return r * t;
}

__global__ void k_finalize(DevBatch b, int mode) {
  chain_wait();
  int sim = blockIdx.x * blockDim.x + threadIdx.x;
  if (sim >= b.nsims) return;
  const SimDev& s = b.sims[sim];
  SimDyn& d = b.dyn[sim];
  unsigned long long bits = d.dtmin_bits;
  double dtmin_cfl = (bits == 0x7FF0000000000000ull) ? kMaxPositive : __longlong_as_double((long long)bits);
  d.dtmin_bits = 0x7FF0000000000000ull;
  if (mode == 0) {
    d.dt_average = 0.0;
    tsd_close(s, d, dtmin_cfl, -999);
    double dt_ic = d.dt;
    tsd_close(s, d, dtmin_cfl, 1);
    d.dt_prev = dt_ic;
    d.step = 0;
    d.time = 0.0;
    d.frozen = 0;
  } else {
    if (d.frozen) return;
    d.time = d.time + d.dt;
    d.step = d.step + 1;
    double dt_cur = d.dt;
    tsd_close(s, d, dtmin_cfl, d.step + 1);
    d.dt_prev = dt_cur;
    if (d.t_end > 0.0 && d.time >= d.t_end) d.frozen = 1;
    // a simulation with a fatal status stops advancing; the others of its
    // batch go on (its segment, cells and boundary quota are its own)
    if (d.status != 0) d.frozen = 1;
  }
  d.dtvel = 0.5 * (d.dt + d.dt_prev);
  // body force of the next step, taken at that step's end time d.time + d.dt
  // (the simulation time when its momentum equation is evaluated): gravity,
  // plus the lateral forcing of a tank moving as x = A sin(w t) seen in the
  // tank frame, A w^2 sin(w t) along x (no reference counterpart; zero
  // amplitude leaves grav unchanged)
  d.geff[0] = s.forcing_aw2 != 0.0 ? s.grav[0] + s.forcing_aw2 * forcing_sin(s.forcing_w * (d.time + d.dt))
                                   : s.grav[0];
  d.geff[1] = s.grav[1];
  d.geff[2] = s.grav[2];
}

// sph_set_time_step: the next step's dt set from outside (the minimum over
// the slabs of a decomposed simulation, each of which closed its step with
// the minimum over its own particles).  With pesodt = 0 the closing's dt is
// that minimum itself, so the whole simulation's dt is the minimum of the
// slabs'; before the first step the IC's dt (dt_prev) is the same value.
// dtvel and the next step's body force follow from it as in k_finalize.
__global__ void k_set_dt(DevBatch b, double dt) {
  const int sim = blockIdx.x * blockDim.x + threadIdx.x;
  if (sim >= b.nsims) return;
  const SimDev& s = b.sims[sim];
  SimDyn& d = b.dyn[sim];
  d.dt = dt;
  if (d.step == 0) d.dt_prev = dt;
  d.dtvel = 0.5 * (d.dt + d.dt_prev);
  d.geff[0] = s.forcing_aw2 != 0.0 ? s.grav[0] + s.forcing_aw2 * forcing_sin(s.forcing_w * (d.time + d.dt))
                                   : s.grav[0];
}

// sph_set_clock: the clock of a resumed simulation (sim 0), with dtvel and
// the next step's body force as k_finalize leaves them.
__global__ void k_set_clock(DevBatch b, double time, int step, double dt, double dt_prev, double dt_average) {
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  const SimDev& s = b.sims[0];
  SimDyn& d = b.dyn[0];
  d.time = time;
  d.step = step;
  d.dt = dt;
  d.dt_prev = dt_prev;
  d.dt_average = dt_average;
  d.dtvel = 0.5 * (d.dt + d.dt_prev);
  d.geff[0] = s.forcing_aw2 != 0.0 ? s.grav[0] + s.forcing_aw2 * forcing_sin(s.forcing_w * (d.time + d.dt))
                                   : s.grav[0];
}

// The laminar flags of a resumed simulation, from caller order.
__global__ void k_load_laminar(DevBatch b, const int* flags) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    P.L[p] = (uint8_t)(flags[(size_t)s.p_off + P.I[p] - 1] != 0);
  }
}

// sph_batch_cancel: a simulation still advancing stops from the next launch
// on, with status SPH_CANCELLED; one already frozen (finished or failed)
// keeps its status.
__global__ void k_cancel(DevBatch b, int sim) {
  if (threadIdx.x == 0 && sim < b.nsims && !b.dyn[sim].frozen) {
    atomicCAS(&b.dyn[sim].status, 0, SPH_CANCELLED);
    b.dyn[sim].frozen = 1;
  }
}

// A boundary pass that no sort has just preceded (the per-call ABI).
__global__ void k_bdt_reset(DevBatch b) {
  int sim = blockIdx.x * blockDim.x + threadIdx.x;
  if (sim < b.nsims) reset_boundary_counters(b, sim);
}

// ==========================================================================
// Global quantities (fluid_global_quantities.f90:59-72): FP64 sums over the
// fluid of mass, linear momentum, angular momentum about the origin
// (Vector_Product.f90 of coord and vel) and volume m / rho.  The reference
// sums sequentially in pg order; here each tile's particles are summed by a
// fixed shuffle tree and the tiles of a simulation in tile order, every
// addition compensated (a sum and its rounding error), so the result is the
// exact sum up to a few ulps and does not depend on the launch shape.
// ==========================================================================
struct CSum {
  double s, c;   // sum, accumulated rounding error
};

// TwoSum (Knuth) of the leading parts, the trailing parts added, then
// renormalised so |c| stays below an ulp of s.
__device__ __forceinline__ CSum csum_add(CSum a, CSum b) {
  const double s = a.s + b.s;
  const double bb = s - a.s;
  const double e = (a.s - (s - bb)) + (b.s - bb);
  const double c = (a.c + b.c) + e;
  const double t = s + c;
  return CSum{t, c - (t - s)};
}

__device__ __forceinline__ CSum csum_warp(CSum a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    CSum b{__shfl_down_sync(0xffffffffu, a.s, o), __shfl_down_sync(0xffffffffu, a.c, o)};
    a = csum_add(a, b);
  }
  return a;
}

constexpr int kGlobalQ = 8;

// Per-tile compensated partial sums: part[t][q] = (s, c).
__global__ void __launch_bounds__(kBlock) k_global_partials(DevBatch b, double2* part) {
  __shared__ SimDev s;
  __shared__ CSum ws[kBlock / 32][kGlobalQ];
  int cur = -1;
  const Particles& P = b.P;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    const int p = tl.start + threadIdx.x;
    double q[kGlobalQ];
#pragma unroll
    for (int k = 0; k < kGlobalQ; ++k) q[k] = 0.0;
    if (threadIdx.x < tl.count && p < s.p_off + b.dyn[tl.sim].nag) {
      const double4 x = P.X[p];
      const double4 u = P.V[p];
      const double m = x.w;
      q[0] = m;
      q[1] = m * u.x;
      q[2] = m * u.y;
      q[3] = m * u.z;
      q[4] = m * (x.y * u.z - x.z * u.y);
      q[5] = m * (x.z * u.x - x.x * u.z);
      q[6] = m * (x.x * u.y - x.y * u.x);
      q[7] = m / P.RP[p].x;
    }
#pragma unroll
    for (int k = 0; k < kGlobalQ; ++k) {
      CSum a = csum_warp(CSum{q[k], 0.0});
      if (lane == 0) ws[warp][k] = a;
    }
    __syncthreads();
    if (threadIdx.x < kGlobalQ) {
      CSum a = ws[0][threadIdx.x];
      for (int w = 1; w < kBlock / 32; ++w) a = csum_add(a, ws[w][threadIdx.x]);
      part[(size_t)t * kGlobalQ + threadIdx.x] = make_double2(a.s, a.c);
    }
    __syncthreads();
  }
}

// One warp per simulation: its tiles' partials in tile order (lane l takes
// tiles l, l + 32, ...), then the fixed shuffle tree.
__global__ void k_global_final(DevBatch b, const double2* __restrict__ part, double* out) {
  const int sim = blockIdx.x;
  const int lane = threadIdx.x;
  const int t0 = b.sims[sim].p_off / kBlock;
  const int t1 = t0 + (b.sims[sim].cap + kBlock - 1) / kBlock;
  for (int k = 0; k < kGlobalQ; ++k) {
    CSum a{0.0, 0.0};
    for (int t = t0 + lane; t < t1; t += 32) {
      const double2 v = part[(size_t)t * kGlobalQ + k];
      a = csum_add(a, CSum{v.x, v.y});
    }
    a = csum_warp(a);
    if (lane == 0) out[(size_t)sim * kGlobalQ + k] = a.s + a.c;
  }
}

// ==========================================================================
// Caller-order transfer and verification dumps
// ==========================================================================
__global__ void k_init_from_caller(DevBatch b, const double* x, const double* v, const double* rho, const double* p,
                                   const double* m) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    if (threadIdx.x >= tl.count) continue;
    int q = tl.start + threadIdx.x;           // caller order slot
    int i = q - s.p_off;                       // caller index - 1
    if (i < b.dyn[tl.sim].nag) {
      P.X2[q] = make_double4(x[3 * (size_t)q], x[3 * (size_t)q + 1], x[3 * (size_t)q + 2], m[q]);
      P.V2[q] = make_double4(v[3 * (size_t)q], v[3 * (size_t)q + 1], v[3 * (size_t)q + 2], rho[q]);
      P.P2[q] = p[q];
      P.I2[q] = i + 1;
    } else {
      P.X2[q] = make_double4(0, 0, 0, 0);
      P.V2[q] = make_double4(0, 0, 0, 1.0);
      P.P2[q] = 0.0;
      P.I2[q] = 0;
    }
    P.L2[q] = 0;
  }
}

// k_init_from_caller in two halves, for an upload whose positions and
// masses arrive first: the positions half also marks each slot's caller
// index (0 = empty), and the rest half fills a slot's velocity, density and
// pressure where that mark is set.  The rest half does not read the particle
// count, which the removal pass of the concurrent sort may be lowering.
__global__ void k_init_positions(DevBatch b, const double* x, const double* m) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    if (threadIdx.x >= tl.count) continue;
    int q = tl.start + threadIdx.x;
    int i = q - s.p_off;
    if (i < b.dyn[tl.sim].nag) {
      P.X2[q] = make_double4(x[3 * (size_t)q], x[3 * (size_t)q + 1], x[3 * (size_t)q + 2], m[q]);
      P.I2[q] = i + 1;
    } else {
      P.X2[q] = make_double4(0, 0, 0, 0);
      P.I2[q] = 0;
    }
    P.L2[q] = 0;
  }
}

__global__ void k_init_rest(DevBatch b, const double* v, const double* rho, const double* p) {
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    if (threadIdx.x >= tl.count) continue;
    int q = tl.start + threadIdx.x;
    if (P.I2[q] != 0) {
      P.V2[q] = make_double4(v[3 * (size_t)q], v[3 * (size_t)q + 1], v[3 * (size_t)q + 2], rho[q]);
      P.P2[q] = p[q];
    } else {
      P.V2[q] = make_double4(0, 0, 0, 1.0);
      P.P2[q] = 0.0;
    }
  }
}

__global__ void k_to_caller(DevBatch b, double* x, double* v, double* rho, double* p, double* m, double* acc,
                            double* dden) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int q = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || q >= s.p_off + b.dyn[tl.sim].nag) continue;
    size_t o = (size_t)s.p_off + P.I[q] - 1;
    double4 xx = P.X[q];
    double4 vv = P.V[q];
    double2 rp = P.RP[q];
    if (x) { x[3 * o] = xx.x; x[3 * o + 1] = xx.y; x[3 * o + 2] = xx.z; }
    if (v) { v[3 * o] = vv.x; v[3 * o + 1] = vv.y; v[3 * o + 2] = vv.z; }
    if (rho) rho[o] = rp.x;
    if (p) p[o] = rp.y;
    if (m) m[o] = xx.w;
    if (acc) { double4 a = P.ACC[q]; acc[3 * o] = a.x; acc[3 * o + 1] = a.y; acc[3 * o + 2] = a.z; }
    if (dden) dden[o] = P.DDEN[q];
  }
}

// Positions, velocities and masses of a fused step's record (X2, V2, I2 in
// the last sort's slot order, written by the momentum pass and final from
// then on) to caller order, before the step's own sort has run.  Slots are
// those below the particle count; the sort's removal pass may lower that
// count concurrently, in which case the caller redoes this copy from the
// sorted state (the removal renumbers particles).
__global__ void k_scratch_to_caller(DevBatch b, double* x, double* v, double* m) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int q = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || q >= s.p_off + b.dyn[tl.sim].nag) continue;
    const int id = P.I2[q];
    if (id <= 0) continue;
    const size_t o = (size_t)s.p_off + id - 1;
    const double4 xx = P.X2[q];
    const double4 vv = P.V2[q];
    x[3 * o] = xx.x; x[3 * o + 1] = xx.y; x[3 * o + 2] = xx.z;
    v[3 * o] = vv.x; v[3 * o + 1] = vv.y; v[3 * o + 2] = vv.z;
    m[o] = xx.w;
  }
}

template <int DIM>
__global__ void k_dump_neighbours(DevBatch b, int nmaxj, int* counts, int* lists) {
  // the stored lists the pair passes read, in caller indices, with the
  // particle itself put back where the reference's visiting order has it
  // (the lists leave it out): before the first entry past its own slot in
  // its own column (the centre run).  It was accepted unless the NMAXPARTJ
  // cap cut the list before it, in which case cnt reached the cap.
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  constexpr unsigned kCentre = (DIM == 3) ? 4u : 1u;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    size_t row = (size_t)s.p_off + P.I[p] - 1;
    const int cnt = b.ncount[p];
    const int* base = reinterpret_cast<const int*>(reinterpret_cast<const int4*>(b.nlist) + list_base4(p, b.list_cap4));
    bool self = cnt < s.nmaxpartj;
    int n = 0;
    for (int k = 0; k < cnt; ++k) {
      const unsigned e = (unsigned)base[(size_t)(k >> 2) * 128 + (k & 3)];
      const unsigned run = e >> kSlotBits;
      const int q = (int)(e & kSlotMask);
      if (self && (run > kCentre || (run == kCentre && q > p))) {
        if (n < nmaxj) lists[row * nmaxj + n] = P.I[p];
        n++;
        self = false;
      }
      if (n < nmaxj) lists[row * nmaxj + n] = P.I[q];
      n++;
    }
    if (self) {
      if (n < nmaxj) lists[row * nmaxj + n] = P.I[p];
      n++;
    }
    counts[row] = n;
  }
}

__global__ void k_dump_boundary(DevBatch b, int max_per, int* ncb, int* clob, double* vals) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    size_t row = (size_t)s.p_off + P.I[p] - 1;
    int n = P.bdt_count[p];
    ncb[row] = n;
    for (int k = 0; k < n && k < max_per; ++k) {
      const BdtEntry& e = P.bdt[P.bdt_start[p] + k];
      clob[row * max_per + k] = e.clobonum;
      double* d = vals + (row * max_per + k) * 20;
      for (int q = 0; q < 3; ++q) d[q] = e.loc[q];
      for (int q = 0; q < 8; ++q) d[3 + q] = e.bi[q];
      // IntGiWrRdV(3,3) column-major
      for (int c = 0; c < 3; ++c)
        for (int r = 0; r < 3; ++r) d[11 + 3 * c + r] = e.ig[3 * r + c];
    }
  }
}

// B_ren_gradp / B_ren_divu by caller index, B(i,j) at [9 row + 3 i + j].
__global__ void k_dump_renormalisation(DevBatch b, double* bg, double* bd) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    size_t row = (size_t)s.p_off + P.I[p] - 1;
    for (int k = 0; k < 9; ++k) {
      if (bg && P.BG) bg[9 * row + k] = P.BG[(size_t)k * P.total_slots + p];
      if (bd && P.BD) bd[9 * row + k] = P.BD[(size_t)k * P.total_slots + p];
    }
  }
}

__global__ void k_dump_cella(DevBatch b, int* cella) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    double4 xi = P.X[p];
    int i, j, k;
    int c = 0;
    if (particle_cell(s, xi.x, xi.y, xi.z, i, j, k)) c = ((k - 1) * s.ncd[1] + (j - 1)) * s.ncd[0] + i;
    cella[(size_t)s.p_off + P.I[p] - 1] = c;
  }
}

// pg%laminar_flag (inter_EqMoto.f90:269-283) of the last momentum pass, in
// caller order.
__global__ void k_dump_laminar(DevBatch b, int* flags) {
  __shared__ SimDev s;
  int cur = -1;
  const Particles& P = b.P;
  for (int t = blockIdx.x; t < b.ntiles; t += gridDim.x) {
    Tile tl = b.tiles[t];
    load_sim(s, b.sims, tl.sim, cur);
    int p = tl.start + threadIdx.x;
    if (threadIdx.x >= tl.count || p >= s.p_off + b.dyn[tl.sim].nag) continue;
    flags[(size_t)s.p_off + P.I[p] - 1] = P.L[p];
  }
}

// FP64 fused multiply-add throughput probe (8 independent chains per thread).
__global__ void __launch_bounds__(256) k_fp64_probe(double* sink, int iters) {
  double a0 = threadIdx.x * 1e-9, a1 = a0 + 1e-9, a2 = a0 + 2e-9, a3 = a0 + 3e-9;
  double a4 = a0 + 4e-9, a5 = a0 + 5e-9, a6 = a0 + 6e-9, a7 = a0 + 7e-9;
  const double m = 0.999999999, c = 1e-12;
  for (int i = 0; i < iters; ++i) {
    a0 = fma(a0, m, c); a1 = fma(a1, m, c); a2 = fma(a2, m, c); a3 = fma(a3, m, c);
    a4 = fma(a4, m, c); a5 = fma(a5, m, c); a6 = fma(a6, m, c); a7 = fma(a7, m, c);
  }
  double r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (r == 12345.0) sink[blockIdx.x] = r;
}

// FP32 fused multiply-add throughput probe.
__global__ void __launch_bounds__(256) k_fp32_probe(float* sink, int iters) {
  float a0 = threadIdx.x * 1e-6f, a1 = a0 + 1e-6f, a2 = a0 + 2e-6f, a3 = a0 + 3e-6f;
  float a4 = a0 + 4e-6f, a5 = a0 + 5e-6f, a6 = a0 + 6e-6f, a7 = a0 + 7e-6f;
  const float m = 0.9999f, c = 1e-7f;
  for (int i = 0; i < iters; ++i) {
    a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c); a3 = fmaf(a3, m, c);
    a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c); a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
  }
  float r = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (r == 12345.0f) sink[blockIdx.x] = r;
}

double launch_fp32_probe(float* sink, int blocks, cudaStream_t st) {
  const int iters = 8192;
  k_fp32_probe<<<blocks, 256, 0, st>>>(sink, iters);
  return 2.0 * 8.0 * iters * 256.0 * blocks;
}

double launch_fp64_probe(double* sink, int blocks, cudaStream_t st) {
  const int iters = 4096;
  k_fp64_probe<<<blocks, 256, 0, st>>>(sink, iters);
  return 2.0 * 8.0 * iters * 256.0 * blocks;
}

// Self-check of div_rn and of div_rn_unsigned0 against the IEEE division a / b
// (for the latter +0 where a is -0 and b positive) on generated operands
// (SplitMix64 of the seed and the operand index).  Five kinds, by
// index mod 5: random signs, significands and exponents in [-64, 63];
// divisors whose significands are within 255 units of all ones; quotients
// within a few units of 2^-106 relative of a rounding midpoint of a random
// quotient (a = RN(b q + b ulp(q)/2)); a zero dividend of either sign; and
// the ranges of the kernels' operands (1e-6 to 1e3 over 1e-3 to 2e3).
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long z) {
  z += 0x9e3779b97f4a7c15ull;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ double compose_double(unsigned long long frac, int exp, unsigned sign) {
  const unsigned long long bits = ((unsigned long long)(sign & 1u) << 63) |
                                  ((unsigned long long)(exp + 1023) << 52) | (frac & ((1ull << 52) - 1));
  return __longlong_as_double((long long)bits);
}

// bad[0] counts mismatches, bad[1] flags that first[] holds one's operands.
__global__ void __launch_bounds__(256) k_check_division(unsigned long long n, unsigned long long seed,
                                                        unsigned long long* bad, double* first) {
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  unsigned long long nbad = 0;
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const unsigned long long u1 = splitmix64(seed ^ (2 * i)), u2 = splitmix64(seed ^ (2 * i + 1));
    const int e1 = (int)((u1 >> 52) & 127) - 64, e2 = (int)((u2 >> 52) & 127) - 64;
    double a, b;
    switch ((int)(i % 5)) {
      case 0:
        a = compose_double(u1, e1, (unsigned)(u1 >> 63));
        b = compose_double(u2, e2, (unsigned)(u2 >> 63));
        break;
      case 1:
        a = compose_double(u1, e1, (unsigned)(u1 >> 63));
        b = compose_double(((1ull << 52) - 1) - (u2 & 255), e2 & 15, (unsigned)(u2 >> 63));
        break;
      case 2: {
        const double q = compose_double(u1, e1 & 31, 0);
        const double half_ulp = compose_double(0, (e1 & 31) - 53, 0);
        b = compose_double(u2, e2 & 31, (unsigned)(u2 >> 63));
        a = __fma_rn(b, half_ulp, __dmul_rn(b, q));
        break;
      }
      case 3:
        a = (u1 & 1) ? -0.0 : 0.0;
        b = compose_double(u2, e2, (unsigned)(u2 >> 63));
        break;
      default:
        a = compose_double(u1, (int)((u1 >> 52) % 30) - 20, (unsigned)(u1 >> 63));
        b = compose_double(u2, (int)((u2 >> 52) % 21) - 10, 0);
        break;
    }
    const double ref = a / b;
    const double y = __drcp_rn(b);
    const double ref0 = a == 0.0 && b > 0.0 ? 0.0 : ref;
    if (__double_as_longlong(ref) != __double_as_longlong(div_rn(a, b, y)) ||
        __double_as_longlong(ref0) != __double_as_longlong(div_rn_unsigned0(a, b, y))) {
      ++nbad;
      if (atomicCAS(bad + 1, 0ull, 1ull) == 0ull) {   // the first mismatch found keeps its operands
        first[0] = a;
        first[1] = b;
      }
    }
  }
  if (nbad) atomicAdd(bad, nbad);
}

void launch_check_division(unsigned long long n, unsigned long long seed, unsigned long long* bad, double* first,
                           int blocks, cudaStream_t st) {
  k_check_division<<<blocks, 256, 0, st>>>(n, seed, bad, first);
}

// ==========================================================================
// launch wrappers
// ==========================================================================
// A launch that follows the previous one of its stream by programmatic
// dependence (chain_wait), which hides its start-up: about 1.5 us of each gap
// between the step's launches (2D column of 5,000 particles in FP64 2.46 -> 2.41 ms
// for 40 steps, 3D dam break of 13,500 2.35 -> 2.28 for 20, of 256,000 in FP64
// 8.01 -> 7.90 for 10).  No kernel triggers early: blocks that wait on an SM take the
// place of running ones (13,500 particles 10% slower).  From 32 tiles of 256
// particles an SM on the gaps are nothing and ordinary launches the better ones
// (1.14 10^6 particles 0.7% faster so, 8 10^6 1.4% slower).  Launches that follow
// a wait for another stream stay ordinary.
template <typename... P, typename... A>
static void launch_next(void (*kernel)(DevBatch, P...), int grid, int block, cudaStream_t st, const DevBatch& b, A... args) {
  cudaLaunchConfig_t c = {};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.stream = st;
  cudaLaunchAttribute follow = {};
  follow.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  follow.val.programmaticStreamSerializationAllowed = b.ntiles < 32 * b.sms ? 1 : 0;
  c.attrs = &follow;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, kernel, b, P(args)...);
}

static inline int blocks_for(const DevBatch& b) { return b.ntiles < b.grid_blocks ? b.ntiles : b.grid_blocks; }
// The pair and list passes take one block to a tile unless a grid has been
// chosen: they load little per block, and tiles handed out as blocks finish
// even out what a fixed stride of 8 blocks an SM leaves uneven (FP32c box of
// 10^6, lean momentum loop: 528 us so strided, 483 one to a tile).  So does the
// wall pass of the FP64 form (64 2D columns, 1.1 10^6 particles: 882 us a step,
// 891 strided).  That of the FP32c form, beside the lists and the pair sums,
// strides 8 blocks an SM: it is not what the step waits for, and a block that
// stays costs them less than many that come and go (2D column of 1.02 10^6: 490 us a step
// one to a tile, 481 strided; 2.47 10^6: 1089 and 1082; 64 2D columns: 598 and 592;
// 256: 2283 and 2270; 3D dam break of 4 10^6: 5302 and 5286).
static inline int blocks_for(const DevBatch& b, int cls) {
  int g = b.grid[cls];
  if (g <= 0) g = cls == kGridBoundary && b.fp32c ? b.grid_blocks : b.ntiles;
  return b.ntiles < g ? b.ntiles : g;
}

void launch_stage(const DevBatch& b, cudaStream_t st) { k_stage<<<blocks_for(b), kBlock, 0, st>>>(b); }

void launch_bin(const DevBatch& b, KeyKind kind, cudaStream_t st) {
  if (kind == KeyKind::Sort) launch_next(k_bin<KeyKind::Sort>, blocks_for(b), kBlock, st, b);
  else launch_next(k_bin<KeyKind::Reference>, blocks_for(b), kBlock, st, b);
}

void launch_scan(const DevBatch& b, int* cell_start, bool removals, cudaStream_t st) {
  const int n = b.P.total_cells, nb = (n + kScanChunk - 1) / kScanChunk;
  const bool summed = nb > kMostOwnSums;
  if (summed) k_scan_sums<<<1, kScanThreads, 0, st>>>(b.scan_block_sums, nb);
  launch_next(k_scan, nb + (removals ? b.nsims : 0), kScanThreads, st, b, n, nb, cell_start, removals ? 1 : 0,
              summed ? 1 : 0);
}

void launch_cancel(const DevBatch& b, int sim, cudaStream_t st) { k_cancel<<<1, 32, 0, st>>>(b, sim); }

void launch_load_laminar(const DevBatch& b, const int* laminar, cudaStream_t st) {
  k_load_laminar<<<blocks_for(b), kBlock, 0, st>>>(b, laminar);
}
void launch_set_clock(const DevBatch& b, double time, int step, double dt, double dt_prev, double dt_average,
                      const int* laminar, cudaStream_t st) {
  k_set_clock<<<1, 32, 0, st>>>(b, time, step, dt, dt_prev, dt_average);
  if (laminar) launch_load_laminar(b, laminar, st);
}
void launch_set_dt(const DevBatch& b, double dt, cudaStream_t st) {
  k_set_dt<<<(b.nsims + 127) / 128, 128, 0, st>>>(b, dt);
}

void upload_bit2d(const double* tab, cudaStream_t st) {
  cudaMemcpyToSymbolAsync(c_bit2d, tab, sizeof(double) * 22 * 6, 0, cudaMemcpyHostToDevice, st);
}

void launch_place(const DevBatch& b, bool boundary_follows, cudaStream_t st) {
  launch_next(k_place, blocks_for(b), kBlock, st, b, b.P.cell_start, 1, boundary_follows ? 1 : 0);
}

void launch_rank_permute(const DevBatch& b, cudaStream_t st) {
  launch_next(k_rank_permute<kPermuteAll>, blocks_for(b), kBlock, st, b);
}

void launch_rank_permute_positions(const DevBatch& b, cudaStream_t st) {
  launch_next(k_rank_permute<kPermutePositions>, blocks_for(b), kBlock, st, b);
}

void launch_rank_permute_rest(const DevBatch& b, cudaStream_t st) {
  k_rank_permute<kPermuteRest><<<blocks_for(b), kBlock, 0, st>>>(b);
}

void launch_rank_reference(const DevBatch& b, const int* cell_start_ref, int* npartord, cudaStream_t st) {
  launch_next(k_place, blocks_for(b), kBlock, st, b, cell_start_ref, 0, 0);
  k_rank_reference<<<blocks_for(b), kBlock, 0, st>>>(b, cell_start_ref, npartord);
}

void launch_boundary_reset(const DevBatch& b, cudaStream_t st) {
  k_bdt_reset<<<(b.nsims + 127) / 128, 128, 0, st>>>(b);
}

void launch_boundary(const DevBatch& b, cudaStream_t st) {
  if (b.dim == 3) {
    k_boundary3d<<<blocks_for(b, kGridBoundary), kBlock, 0, st>>>(b);
    launch_next(k_boundary3d_integrals, b.grid[kGridIntegrals] > 0 ? b.grid[kGridIntegrals] : b.grid_blocks, 128, st, b);
  } else {
    // a chosen grid counts blocks of kBlock threads, as for the other passes
    const int g = blocks_for(b, kGridBoundary);
    if (b.ntiles >= (b.fp32c ? 8 : 32) * b.sms) k_boundary2d<128><<<2 * g, 128, 0, st>>>(b);
    else k_boundary2d<kBlock><<<g, kBlock, 0, st>>>(b);
  }
}

// 2D with C1_BE: the frontier terms and inversion of the matrices (their
// renormalisation is the identity in 2D, see k_c1_frontier_2d)
static void c1_frontier_2d(const DevBatch& b, bool gradp_only, cudaStream_t st) {
  if (b.dim != 2 || !b.c1) return;
  if (gradp_only) k_c1_frontier_2d<true><<<blocks_for(b), kBlock, 0, st>>>(b);
  else k_c1_frontier_2d<false><<<blocks_for(b), kBlock, 0, st>>>(b);
}

// Four lanes to a particle in a pair pass (without C1), while one lane each
// would leave an SM with fewer than so many warps.  One lane takes the same time up to
// about 8 warps an SM (a particle's chain of pairs), four lanes are one wave of
// blocks at first and then two.  FP32c: the lines are the ends of that wave, 2 and 3
// blocks an SM (momentum us one lane / four: 3D 18,513 particles 39.6 / 29.9,
// 23,328 39.9 / 39.9; 2D 15,576 20.9 / 19.5, 21,632 21.5 / 25.4.  Continuity:
// 2D 15,576 17.4 / 15.3, 27,730 17.4 / 17.4, 32,131 17.4 / 19.4), and in 3D, whose
// lists of 78 make the chain longer, two waves still pay for the continuity
// (37,044: 33.2 / 31.7).  FP64 (momentum: 3D 37,044 82.8 / 73.2; 2D 32,131 28.2 /
// 27.8, 33,800 27.8 / 29.1).
bool momentum_split(const DevBatch& b) { return !b.c1 && b.ntiles * (kBlock / 32) < b.sms * (b.fp32c ? 4 : 7); }
bool continuity_split(const DevBatch& b) {
  const int warps = b.fp32c ? (b.dim == 3 ? 8 : 6) : 7;
  return !b.c1 && b.ntiles * (kBlock / 32) < b.sms * warps;
}
static int split_blocks(const DevBatch& b) { return b.ntiles * (kBlock / (kSplitThreads / 4)); }

void launch_momentum(const DevBatch& b, bool fused, cudaStream_t st) {
  int g = blocks_for(b, kGridMomentum);
  c1_frontier_2d(b, true, st);
  if (momentum_split(b)) {
    const int gs = split_blocks(b);
    if (b.dim == 3) {
      if (fused) k_momentum_split<3, true><<<gs, kSplitThreads, 0, st>>>(b);
      else k_momentum_split<3, false><<<gs, kSplitThreads, 0, st>>>(b);
    } else {
      if (fused) k_momentum_split<2, true><<<gs, kSplitThreads, 0, st>>>(b);
      else k_momentum_split<2, false><<<gs, kSplitThreads, 0, st>>>(b);
    }
    return;
  }
  if (b.dim == 3 && b.c1) {
    if (fused) k_momentum<3, true, true><<<g, kBlock, 0, st>>>(b);
    else k_momentum<3, false, true><<<g, kBlock, 0, st>>>(b);
  } else if (b.dim == 3) {
    if (b.mom_batch) {
      if (fused) k_momentum<3, true, false, true><<<g, kBlock, 0, st>>>(b);
      else k_momentum<3, false, false, true><<<g, kBlock, 0, st>>>(b);
    } else {
      if (fused) k_momentum<3, true><<<g, kBlock, 0, st>>>(b);
      else k_momentum<3, false><<<g, kBlock, 0, st>>>(b);
    }
  } else {
    if (b.mom_batch) {
      if (fused) k_momentum<2, true, false, true><<<g, kBlock, 0, st>>>(b);
      else k_momentum<2, false, false, true><<<g, kBlock, 0, st>>>(b);
    } else {
      if (fused) k_momentum<2, true><<<g, kBlock, 0, st>>>(b);
      else k_momentum<2, false><<<g, kBlock, 0, st>>>(b);
    }
  }
}

void launch_neighbour_lists(const DevBatch& b, cudaStream_t st) {
  // a chosen grid counts blocks of kBlock threads, as for the other passes
  const int tiles = b.grid[kGridLists] > 0 && b.grid[kGridLists] < b.ntiles ? b.grid[kGridLists] : b.ntiles;
  const int g = tiles * (kBlock / kListBlock);
  if (b.dim == 3) launch_next(k_neighbour_lists<3>, g, kListBlock, st, b);
  else launch_next(k_neighbour_lists<2>, g, kListBlock, st, b);
}

void launch_renormalisation(const DevBatch& b, cudaStream_t st) {
  if (!b.c1) return;
  if (b.dim == 3) k_renormalisation<3><<<blocks_for(b, kGridLists), kBlock, 0, st>>>(b);
  else k_renormalisation<2><<<blocks_for(b, kGridLists), kBlock, 0, st>>>(b);
}

void launch_momentum_f32(const DevBatch& b, bool fused, cudaStream_t st) {
  int g = blocks_for(b, kGridMomentum);
  int gf = blocks_for(b);
  c1_frontier_2d(b, true, st);
  const int f = fused ? 1 : 0;
  if (b.dim == 3 && b.c1) {
    k_momentum_f32<3, true><<<g, kBlock, 0, st>>>(b, f);
    if (fused) launch_next(k_momentum_f32_finish<3, true, true>, gf, kBlock, st, b);
    else launch_next(k_momentum_f32_finish<3, false, true>, gf, kBlock, st, b);
  } else if (b.dim == 3) {
    if (momentum_split(b)) k_momentum_f32_split<3><<<b.ntiles * 4, kBlock, 0, st>>>(b, f);
    else if (b.mom_batch == 2) k_momentum_f32<3, false, true, true><<<g, kBlock, 0, st>>>(b, f);
    else if (b.mom_batch) k_momentum_f32<3, false, true><<<g, kBlock, 0, st>>>(b, f);
    else k_momentum_f32<3><<<g, kBlock, 0, st>>>(b, f);
    if (fused) launch_next(k_momentum_f32_finish<3, true>, gf, kBlock, st, b);
    else launch_next(k_momentum_f32_finish<3, false>, gf, kBlock, st, b);
  } else {
    if (momentum_split(b)) k_momentum_f32_split<2><<<b.ntiles * 4, kBlock, 0, st>>>(b, f);
    else if (b.mom_batch == 2) k_momentum_f32<2, false, true, true><<<g, kBlock, 0, st>>>(b, f);
    else if (b.mom_batch) k_momentum_f32<2, false, true><<<g, kBlock, 0, st>>>(b, f);
    else k_momentum_f32<2><<<g, kBlock, 0, st>>>(b, f);
    if (fused) launch_next(k_momentum_f32_finish<2, true>, gf, kBlock, st, b);
    else launch_next(k_momentum_f32_finish<2, false>, gf, kBlock, st, b);
  }
}

void launch_continuity_f32_pairs(const DevBatch& b, cudaStream_t st) {
  int g = blocks_for(b, kGridContinuity);
  if (b.dim == 3 && b.c1_divu) launch_next(k_continuity_f32<3, true>, g, kBlock, st, b);
  else if (continuity_split(b) && b.dim == 3) launch_next(k_continuity_f32_split<3>, b.ntiles * 4, kBlock, st, b);
  else if (continuity_split(b)) launch_next(k_continuity_f32_split<2>, b.ntiles * 4, kBlock, st, b);
  else if (b.dim == 3 && b.con_batch == 2) launch_next(k_continuity_f32<3, false, true, true>, g, kBlock, st, b);
  else if (b.dim == 3 && b.con_batch) launch_next(k_continuity_f32<3, false, true>, g, kBlock, st, b);
  else if (b.dim == 3) launch_next(k_continuity_f32<3>, g, kBlock, st, b);
  else if (b.con_batch == 2) launch_next(k_continuity_f32<2, false, true, true>, g, kBlock, st, b);
  else if (b.con_batch) launch_next(k_continuity_f32<2, false, true>, g, kBlock, st, b);
  else launch_next(k_continuity_f32<2>, g, kBlock, st, b);
}

void launch_continuity_f32_finish(const DevBatch& b, bool fused, cudaStream_t st) {
  int g = blocks_for(b);
  c1_frontier_2d(b, false, st);
  if (b.dim == 3 && b.c1) {
    if (fused) k_continuity_f32_finish<3, true, true><<<g, kBlock, 0, st>>>(b);
    else k_continuity_f32_finish<3, false, true><<<g, kBlock, 0, st>>>(b);
  } else if (b.dim == 3) {
    if (fused) k_continuity_f32_finish<3, true><<<g, kBlock, 0, st>>>(b);
    else k_continuity_f32_finish<3, false><<<g, kBlock, 0, st>>>(b);
  } else {
    if (fused) k_continuity_f32_finish<2, true><<<g, kBlock, 0, st>>>(b);
    else k_continuity_f32_finish<2, false><<<g, kBlock, 0, st>>>(b);
  }
}

void launch_continuity_f32(const DevBatch& b, bool fused, cudaStream_t st) {
  launch_continuity_f32_pairs(b, st);
  launch_continuity_f32_finish(b, fused, st);
}

void launch_refresh_f32(const DevBatch& b, cudaStream_t st) { k_refresh_f32<<<blocks_for(b), kBlock, 0, st>>>(b); }

void launch_continuity(const DevBatch& b, bool fused, cudaStream_t st) {
  int g = blocks_for(b, kGridContinuity);
  c1_frontier_2d(b, false, st);
  if (continuity_split(b)) {
    const int gs = split_blocks(b);
    if (b.dim == 3) {
      if (fused) k_continuity_split<3, true><<<gs, kSplitThreads, 0, st>>>(b);
      else k_continuity_split<3, false><<<gs, kSplitThreads, 0, st>>>(b);
    } else {
      if (fused) k_continuity_split<2, true><<<gs, kSplitThreads, 0, st>>>(b);
      else k_continuity_split<2, false><<<gs, kSplitThreads, 0, st>>>(b);
    }
    return;
  }
  if (b.dim == 3 && b.c1) {
    if (fused) k_continuity<3, true, true><<<g, kBlock, 0, st>>>(b);
    else k_continuity<3, false, true><<<g, kBlock, 0, st>>>(b);
  } else if (b.dim == 3) {
    if (b.con_batch) {
      if (fused) k_continuity<3, true, false, true><<<g, kBlock, 0, st>>>(b);
      else k_continuity<3, false, false, true><<<g, kBlock, 0, st>>>(b);
    } else {
      if (fused) k_continuity<3, true><<<g, kBlock, 0, st>>>(b);
      else k_continuity<3, false><<<g, kBlock, 0, st>>>(b);
    }
  } else {
    if (b.con_batch) {
      if (fused) k_continuity<2, true, false, true><<<g, kBlock, 0, st>>>(b);
      else k_continuity<2, false, false, true><<<g, kBlock, 0, st>>>(b);
    } else {
      if (fused) k_continuity<2, true><<<g, kBlock, 0, st>>>(b);
      else k_continuity<2, false><<<g, kBlock, 0, st>>>(b);
    }
  }
}

void launch_leapfrog_momentum(const DevBatch& b, cudaStream_t st) {
  k_leapfrog_momentum<<<blocks_for(b), kBlock, 0, st>>>(b);
}
void launch_leapfrog_trajectories(const DevBatch& b, cudaStream_t st) {
  k_leapfrog_trajectories<<<blocks_for(b), kBlock, 0, st>>>(b);
}
void launch_leapfrog_continuity(const DevBatch& b, cudaStream_t st) {
  k_leapfrog_continuity<<<blocks_for(b), kBlock, 0, st>>>(b);
}
void launch_eos(const DevBatch& b, cudaStream_t st) { k_eos<<<blocks_for(b), kBlock, 0, st>>>(b); }

void launch_velocity_smoothing(const DevBatch& b, bool fused, bool fp32c, cudaStream_t st) {
  const double4* vel = fused ? b.P.V2 : b.P.V;
  if (fp32c) {
    if (b.dim == 3) launch_next(k_velocity_smoothing_f32<3>, blocks_for(b), kBlock, st, b, vel);
    else launch_next(k_velocity_smoothing_f32<2>, blocks_for(b), kBlock, st, b, vel);
  } else {
    if (b.dim == 3) launch_next(k_velocity_smoothing<3>, blocks_for(b), kBlock, st, b, vel);
    else launch_next(k_velocity_smoothing<2>, blocks_for(b), kBlock, st, b, vel);
  }
  if (fused) launch_next(k_velocity_smoothing_apply<true>, blocks_for(b), kBlock, st, b);
  else launch_next(k_velocity_smoothing_apply<false>, blocks_for(b), kBlock, st, b);
}

void launch_pressure_smoothing(const DevBatch& b, bool fp32c, cudaStream_t st) {
  const bool refresh_f32 = fp32c;
  if (fp32c) {
    if (b.dim == 3) launch_next(k_pressure_smoothing_f32<3>, blocks_for(b), kBlock, st, b);
    else launch_next(k_pressure_smoothing_f32<2>, blocks_for(b), kBlock, st, b);
  } else {
    if (b.dim == 3) launch_next(k_pressure_smoothing<3>, blocks_for(b), kBlock, st, b);
    else launch_next(k_pressure_smoothing<2>, blocks_for(b), kBlock, st, b);
  }
  launch_next(k_pressure_smoothing_apply, blocks_for(b), kBlock, st, b, refresh_f32 ? 1 : 0);
}
void launch_dt_reduce(const DevBatch& b, cudaStream_t st) { k_dt_reduce<<<blocks_for(b), kBlock, 0, st>>>(b); }
void launch_finalize(const DevBatch& b, int mode, cudaStream_t st) {
  launch_next(k_finalize, (b.nsims + 127) / 128, 128, st, b, mode);
}

void launch_init_from_caller(const DevBatch& b, const double* x, const double* v, const double* rho,
                             const double* p, const double* m, cudaStream_t st) {
  k_init_from_caller<<<blocks_for(b), kBlock, 0, st>>>(b, x, v, rho, p, m);
}
void launch_scratch_to_caller(const DevBatch& b, double* x, double* v, double* m, cudaStream_t st) {
  k_scratch_to_caller<<<blocks_for(b), kBlock, 0, st>>>(b, x, v, m);
}
void launch_init_positions(const DevBatch& b, const double* x, const double* m, cudaStream_t st) {
  k_init_positions<<<blocks_for(b), kBlock, 0, st>>>(b, x, m);
}
void launch_init_rest(const DevBatch& b, const double* v, const double* rho, const double* p, cudaStream_t st) {
  k_init_rest<<<blocks_for(b), kBlock, 0, st>>>(b, v, rho, p);
}
void launch_to_caller(const DevBatch& b, double* x, double* v, double* rho, double* p, double* m, double* acc,
                      double* dden, cudaStream_t st) {
  k_to_caller<<<blocks_for(b), kBlock, 0, st>>>(b, x, v, rho, p, m, acc, dden);
}
void launch_dump_neighbours(const DevBatch& b, int nmaxj, int* counts, int* lists, cudaStream_t st) {
  if (b.dim == 3) k_dump_neighbours<3><<<blocks_for(b), kBlock, 0, st>>>(b, nmaxj, counts, lists);
  else k_dump_neighbours<2><<<blocks_for(b), kBlock, 0, st>>>(b, nmaxj, counts, lists);
}
void launch_dump_boundary(const DevBatch& b, int max_per, int* ncb, int* clob, double* vals, cudaStream_t st) {
  k_dump_boundary<<<blocks_for(b), kBlock, 0, st>>>(b, max_per, ncb, clob, vals);
}
void launch_dump_renormalisation(const DevBatch& b, double* bg, double* bd, cudaStream_t st) {
  k_dump_renormalisation<<<blocks_for(b), kBlock, 0, st>>>(b, bg, bd);
}
void launch_global_quantities(const DevBatch& b, double2* part, double* out, cudaStream_t st) {
  k_global_partials<<<blocks_for(b), kBlock, 0, st>>>(b, part);
  k_global_final<<<b.nsims, 32, 0, st>>>(b, part, out);
}

void launch_dump_cella(const DevBatch& b, int* cella, cudaStream_t st) {
  k_dump_cella<<<blocks_for(b), kBlock, 0, st>>>(b, cella);
}

void launch_dump_laminar(const DevBatch& b, int* flags, cudaStream_t st) {
  k_dump_laminar<<<blocks_for(b), kBlock, 0, st>>>(b, flags);
}

}  // namespace sph
