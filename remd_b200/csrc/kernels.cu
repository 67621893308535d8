// kernels.cu -- device code of the B200 REMD engine.  See kernels.cuh for the
// step decomposition and engine_types.cuh for the data layout.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "integrator.cuh"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace remd {

constexpr int kRepThreads = 256;   // threads of the per-replica kernels
constexpr int kBitmapMaxWords = 64; // list-rebuild bitmap window: 2048 molecules per pass
constexpr int kCellMinPrune = 4;    // cut a replica into cells when they prune at least 4x,
constexpr int kCellMinMol = 512;    // and it is no smaller than this (cell_grid)
constexpr int kGroup = 8;           // FP32 form: lanes per molecule in the list and pair kernels
constexpr int kWarpMol = 32 / kGroup;   // molecules of a warp there
constexpr int kPairWarps = kPart2Mol / kWarpMol;   // warps of a list or pair block (kPart2Mol molecules)
constexpr int kSegPairs = 32 * kGroup;  // pairs of a molecule per FP32 partial sum (32 per lane)

int pack_stride(int nsite, int prec) {
  if (prec == kF32) return ((3 + 3 * nsite) + 3) / 4 * 4;   // words, 16-B multiple
  return ((3 + 3 * nsite) + 1) / 2 * 2;                      // doubles, 16-B multiple
}

PairConst pair_const(const RepConst& c) {
  PairConst p{};
  p.nmol = c.nmol; p.mol_off = c.mol_off; p.nsite = c.nsite; p.part2_off = c.part2_off;
  p.nbr_stride = c.nbr_stride; p.nbr_cap = c.nbr_cap; p.confined = c.confined;
  p.nbr_off = c.nbr_off;
  p.rc = (float)c.rc; p.rs = (float)c.rs; p.rc2 = (float)(c.rc * c.rc); p.coef = (float)c.coef_sw;
  p.sgm2q = (float)(0.25 * c.sgm2); p.eps4 = (float)(4.0 * c.eps); p.reach = (float)c.site_reach;
  p.uu = (float)c.qq[c.c0 + 1][c.c0 + 1];
  for (int k = 0; k < c.nsite; k++)
    for (int l = 0; l < c.nsite; l++) p.qq[k][l] = (float)c.qq[k][l];
  for (int k = 0; k < kMaxSites; k++)
    for (int x = 0; x < 3; x++) p.body[k][x] = c.body[k][x];
  return p;
}

int pair_model(const RepConst& c) {
  const double* q = c.qr;
  const auto is = [&](int k, int l, float ratio) { return (float)(q[k] / q[l]) == ratio; };
  const bool std_q = c.nsite == 3   ? is(0, 1, -2.f) && is(2, 1, 1.f)
                     : c.nsite == 4 ? is(2, 1, 1.f) && is(3, 1, -2.f)
                                    : is(2, 1, 1.f) && is(3, 1, -1.f) && is(4, 1, -1.f);
  return c.nsite + (std_q ? kStdCharges : 0);
}

// ------------------------------------------------------------------ reductions
template <int K>
__device__ inline void block_sum(double* v, double* sm) {
  // deterministic: fixed shuffle tree, then warp partials summed in warp order
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  __syncthreads();
  if (lane == 0)
    for (int k = 0; k < K; k++) sm[warp * K + k] = v[k];
  __syncthreads();
  for (int k = 0; k < K; k++) {
    double t = 0.0;
    for (int w = 0; w < nw; w++) t += sm[w * K + k];
    v[k] = t;
  }
  __syncthreads();
}

__device__ inline double block_max(double v, double* sm) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if (lane == 0) sm[warp] = v;
  __syncthreads();
  double t = 0.0;
  for (int w = 0; w < nw; w++) t = fmax(t, sm[w]);
  __syncthreads();
  return t;
}

// Deterministic warp reductions (fixed xor tree; lane 0's value is used).
template <int K>
__device__ inline void warp_sum(double* v) {
#pragma unroll
  for (int k = 0; k < K; k++)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
}

__device__ inline double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum of the force partials of replica c (ordered pairs -> halved like
// ForceCalculator::Switching, src/force_calculator.cxx:775-778).  Called by
// all 32 lanes of one warp: lane l sums records l, l+32, ..., then a butterfly
// over the lanes.  Every lane ends with the same bits (the two partners of a
// butterfly step add the same two numbers) and the order depends only on the
// replica's record count, so every kernel that needs the sums gets identical
// values.  One warp loads all records at once instead of one thread walking
// them: the per-replica scalar chains of the step kernels start sooner.
struct P2Sum {
  double lj, clmb, wall, vir[3];
};
__device__ inline P2Sum reduce_part2(const DevPtrs& d, int part2_off, int npart2) {
  double v[6] = {0, 0, 0, 0, 0, 0};
  for (int t = part2_off + (threadIdx.x & 31); t < part2_off + npart2; t += 32) {
    const Part2 p = d.part2[t];
    v[0] += p.lj; v[1] += p.clmb; v[2] += p.wall;
    v[3] += p.vir[0]; v[4] += p.vir[1]; v[5] += p.vir[2];
  }
  warp_sum<6>(v);
  P2Sum e;
  e.lj = v[0] * 0.5;
  e.clmb = v[1] * 0.5;
  e.wall = v[2];
  e.vir[0] = v[3] * 0.5; e.vir[1] = v[4] * 0.5; e.vir[2] = v[5] * 0.5;
  return e;
}

// Programmatic dependent launch of the MD-step kernels (launch_integrate_prec,
// launch_force): where a step's pair work is small (DevPtrs::pdl), each is
// launched allowed to start while the kernel before it on its stream is still
// running.  Its blocks first wait for that kernel's completion and memory
// (griddepcontrol.wait, which returns at once when there is no such kernel or
// the launch was a plain one), then let the next kernel be scheduled.  A step
// kernel thus reads nothing of its predecessor early; what overlaps is the
// next launch's scheduling with this kernel's last wave.
__device__ __forceinline__ void step_kernel_entry() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Difference of two fixed-point box fractions with 32-bit wraparound: the
// minimum-image separation in units of L / 2^32 (defined via unsigned arithmetic).
__device__ __forceinline__ int wrap_diff(int a, int b) { return (int)((unsigned)a - (unsigned)b); }

// ------------------------------------------------------------------ force records
__device__ inline int fix_coord(double r) {
  // box fraction in [0,1) -> (r-0.5)*2^32 as a wrapping int32
  return (int)(unsigned int)(long long)llrint((r - 0.5) * kFix);
}

// Rotation matrix (body to space) of a quaternion, the map of body_to_space.
struct Rot {
  double m[3][3];
  __device__ __forceinline__ explicit Rot(const double* a) {
    const double a0 = a[0] * a[0], a1 = a[1] * a[1], a2 = a[2] * a[2], a3 = a[3] * a[3];
    const double a01 = a[0] * a[1], a02 = a[0] * a[2], a03 = a[0] * a[3];
    const double a12 = a[1] * a[2], a13 = a[1] * a[3], a23 = a[2] * a[3];
    m[0][0] = a0 + a1 - a2 - a3; m[0][1] = 2. * (a12 - a03); m[0][2] = 2. * (a13 + a02);
    m[1][0] = 2. * (a12 + a03); m[1][1] = a0 - a1 + a2 - a3; m[1][2] = 2. * (a23 - a01);
    m[2][0] = 2. * (a13 - a02); m[2][1] = 2. * (a23 + a01); m[2][2] = a0 - a1 - a2 + a3;
  }
  __device__ __forceinline__ double at(int x, const double* b) const {
    return m[x][0] * b[0] + m[x][1] * b[1] + m[x][2] * b[2];
  }
};

template <int S>
__device__ __forceinline__ void write_pack_f32(const DevPtrs& d, const RepConst& c, int g, const int* fx,
                                               const double* q) {
  constexpr int NV = ((3 + 3 * S) + 3) / 4;
  uint32_t buf[4 * NV];
  for (int k = 3 + 3 * S; k < 4 * NV; k++) buf[k] = 0u;
  for (int x = 0; x < 3; x++) buf[x] = (uint32_t)fx[x];
  const Rot R(q);
#pragma unroll
  for (int k = 0; k < S; k++)
    for (int x = 0; x < 3; x++) buf[3 + 3 * k + x] = __float_as_uint((float)R.at(x, c.body[k]));
  uint4* w4 = reinterpret_cast<uint4*>(d.pack) + g;
#pragma unroll
  for (int k = 0; k < NV; k++)
    w4[(long long)k * d.N] = make_uint4(buf[4 * k], buf[4 * k + 1], buf[4 * k + 2], buf[4 * k + 3]);
}

// The force record of molecule li at (r, q); fx: its fixed-point centre.
__device__ inline void write_pack(const DevPtrs& d, const RepConst& c, int prec, int li, const double* r,
                                  const double* q, const int* fx) {
  const int ns = c.nsite, g = c.mol_off + li;
  if (prec == kF32) {
    if (ns == 3) write_pack_f32<3>(d, c, g, fx, q);
    else if (ns == 4) write_pack_f32<4>(d, c, g, fx, q);
    else write_pack_f32<5>(d, c, g, fx, q);
  } else {
    double* w = reinterpret_cast<double*>(d.pack) + c.pack_off + (long long)li * c.pack_stride;
    w[0] = r[0]; w[1] = r[1]; w[2] = r[2];
    const Rot R(q);
    for (int k = 0; k < ns; k++)
      for (int x = 0; x < 3; x++) w[3 + 3 * k + x] = R.at(x, c.body[k]);
    // fixed-point centre: the cell of the molecule at the next list build
    d.com[g] = make_int4(fx[0], fx[1], fx[2], 0);
  }
}

__global__ void k_pack(DevPtrs d, int prec) {
  const Tile t = d.tiles[blockIdx.x];
  const RepConst& c = d.rc[t.rep];
  const int i = threadIdx.x;
  if (i < t.count) {
    const int li = t.start + i;
    const int g = c.mol_off + li;
    double r[3], q[4];
    for (int x = 0; x < 3; x++) r[x] = d.r[x * d.N + g];
    for (int x = 0; x < 4; x++) q[x] = d.q[x * d.N + g];
    const int fx[3] = {fix_coord(r[0]), fix_coord(r[1]), fix_coord(r[2])};
    write_pack(d, c, prec, li, r, q, fx);
  }
  if (i == 0) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    d.Lbuild[3 * blockIdx.x] = nan;   // lists must be rebuilt
  }
}

// ------------------------------------------------------------------ integrate
struct StepCoef {
  double coef_v_a[3], coef_p_a;   // end-of-previous-step kick
  double coef_v_c[3], coef_p_c;   // this step's kick
  double coef_xi, coef_r[3];
  double Lb[3];
};

// One MD step's integration.  It is bound by latency, not by throughput (a block's
// FP64 scalar chain, then each molecule's): what a block needs -- the replica's
// constants and scalars, the force partials -- is requested at once from the tile's
// descriptor (14.5 -> 11.8 us a launch at 64 molecules).  CHAIN: one more warp runs the
// scalar chain while the molecules' warps load their state, into registers; for grids
// that leave room for the extra warp (launch_integrate_prec).
template <bool MID, bool CHAIN>
__global__ void __launch_bounds__(CHAIN ? 160 : 128, CHAIN ? 3 : 7)
    k_integrate(DevPtrs d, const RepState* __restrict__ X, RepState* __restrict__ Y, int prec) {
  step_kernel_entry();
  __shared__ StepCoef sc;
  __shared__ std::conditional_t<CHAIN, RepConst, int> own;   // the constants, in shared memory
  const int tix = d.order ? d.order[blockIdx.x] : (int)blockIdx.x;
  const Tile t = d.tiles[tix];
  const int B = blockDim.x, N = d.N;
  const int lead = CHAIN ? B - 32 : 0;                 // first thread of the chain's warp
  const int i = threadIdx.x;
  const bool active = i < t.count;
  const bool chain = i >= lead && i < lead + 32;
  const int g = t.mol_off + t.start + min(i, t.count - 1);
  if constexpr (CHAIN) {
    const uint32_t* cs = reinterpret_cast<const uint32_t*>(d.rc + t.rep);
    for (int k = i; k < (int)(sizeof(RepConst) / 4); k += B) reinterpret_cast<uint32_t*>(&own)[k] = cs[k];
  }
  const RepConst& c = *(CHAIN ? reinterpret_cast<const RepConst*>(&own) : d.rc + t.rep);
  RepState st;
  if (i == lead) {
    st = X[t.rep];
    for (int x = 0; x < 3; x++) sc.Lb[x] = d.Lbuild[3 * tix + x];
  }
  double r[3], v[3], q[4], p[4], f[3], n[4];
  int4 ref;
  auto load_state = [&]() {
    for (int x = 0; x < 3; x++) { r[x] = d.r[x * N + g]; v[x] = d.v[x * N + g]; f[x] = d.f[x * N + g]; }
    for (int x = 0; x < 4; x++) { q[x] = d.q[x * N + g]; p[x] = d.p[x * N + g]; n[x] = d.n[x * N + g]; }
    ref = d.ref_com[g];
  };
  P2Sum e;
  if (chain) e = reduce_part2(d, t.part2_off, t.npart2);
  if (CHAIN && !chain) load_state();
  if (CHAIN) __syncthreads();
  if (i == lead) {
    const double pot = e.lj + e.clmb + e.wall;
    const D5Terms f5 = d5_terms(c, st, pot, e.vir);   // L does not change before the second D5
    if (MID) {   // D5 (scalar) + D6 closing the previous step
      for (int x = 0; x < 3; x++) sc.coef_v_a[x] = st.L[x] * st.s * c.dthalf * c.im;
      sc.coef_p_a = 2.0 * st.s * c.dthalf;
      d5_apply(st, f5);
      d6(c, st);
    }
    d6(c, st);   // D6 opening this step
    for (int x = 0; x < 3; x++) sc.coef_v_c[x] = st.L[x] * st.s * c.dthalf * c.im;
    sc.coef_p_c = 2.0 * st.s * c.dthalf;
    d5_apply(st, f5);
    const double si = 1.0 / st.s;   // D4 leaves s
    sc.coef_xi = 0.25 * si;
    d4(c, st);
    for (int x = 0; x < 3; x++) {
      const double Li = 1.0 / st.L[x];
      sc.coef_r[x] = Li * Li * si * c.dt;
    }
    if (tix == t.tile_off) Y[t.rep] = st;
  }
  __syncthreads();
  if (CHAIN && chain) return;
  if (!CHAIN) load_state();
  double acc[4] = {0, 0, 0, 0};
  double disp = 0.0;
  if (active) {
    const int li = t.start + i;
    if (MID) kick(v, p, q, f, n, sc.coef_v_a, sc.coef_p_a);
    kick(v, p, q, f, n, sc.coef_v_c, sc.coef_p_c);
    const bool T1 = (c.tconstant == 1);
    double sPs = 0.0;
    double xi = rotate(q, p, 3, c.iI[2], sc.coef_xi, c.dthalf);
    if (T1) sPs += 0.5 * xi * xi * c.I[2];
    xi = rotate(q, p, 2, c.iI[1], sc.coef_xi, c.dthalf);
    if (T1) sPs += 0.5 * xi * xi * c.I[1];
    int fx[3];
    for (int x = 0; x < 3; x++) {
      r[x] += v[x] * sc.coef_r[x];
      if (r[x] < 0.0) r[x] += 1.0;
      if (r[x] >= 1.0) r[x] -= 1.0;
      fx[x] = fix_coord(r[x]);
      d.r[x * N + g] = r[x];
      d.v[x * N + g] = v[x];
    }
    xi = rotate(q, p, 1, c.iI[0], sc.coef_xi, c.dt);
    if (c.pconstant > 0 || T1)
      for (int x = 0; x < 3; x++) acc[x] = 2.0 * c.mass * v[x] * v[x];
    if (T1) sPs += xi * xi * c.I[0];
    // displacement since the last neighbour-list build, in the build box
    const double dx = (double)wrap_diff(fx[0], ref.x) * kFixInv * sc.Lb[0];
    const double dy = (double)wrap_diff(fx[1], ref.y) * kFixInv * sc.Lb[1];
    const double dz = (double)wrap_diff(fx[2], ref.z) * kFixInv * sc.Lb[2];
    disp = sqrt(dx * dx + dy * dy + dz * dz);
    if (!(disp == disp)) disp = 1e30;   // NaN box: force a rebuild
    xi = rotate(q, p, 2, c.iI[1], sc.coef_xi, c.dthalf);
    if (T1) sPs += 0.5 * xi * xi * c.I[1];
    xi = rotate(q, p, 3, c.iI[2], sc.coef_xi, c.dthalf);
    if (T1) sPs += 0.5 * xi * xi * c.I[2];
    acc[3] = sPs;
    for (int x = 0; x < 4; x++) { d.q[x * N + g] = q[x]; d.p[x * N + g] = p[x]; }
    write_pack(d, c, prec, li, r, q, fx);
  }
  warp_sum<4>(acc);
  disp = warp_max(disp);
  const int w = (t.start + threadIdx.x) >> 5;   // 32-molecule unit of the replica
  if ((threadIdx.x & 31) == 0 && w < c.nwarp) {
    Part1 pt;
    pt.sum_Pv[0] = acc[0]; pt.sum_Pv[1] = acc[1]; pt.sum_Pv[2] = acc[2];
    pt.sum_Ps = acc[3];
    pt.disp = disp;
    d.part1[c.warp_off + w] = pt;
  }
}

// ------------------------------------------------------------------ force
// Cell of a fixed-point box fraction x = (r - 1/2) 2^32 on an n-cell axis:
// floor(r n), exact (r 2^32 = x + 2^31 as an unsigned word).
__device__ __forceinline__ int cell_coord(int x, int n) {
  const unsigned u = (unsigned)x + 0x80000000u;
  return (int)(((unsigned long long)u * (unsigned)n) >> 32);
}

// Radius the list build tests: rcut + skin widened by the truncation error of its FP32
// test (both forms'), sqrt(3) L_max 2^-16, and a relative 1e-5.
__device__ inline double list_test_radius(const RepConst& c, const double* L) {
  const double lmax = fmax(fmax(L[0], L[1]), L[2]);
  return (c.rc + c.skin + 1.7320508075688772 * lmax * (1.0 / 65536.0)) * (1.0 + 1e-5);
}

// Cells per dimension: as many as fit at least the test radius wide, so that
// every pair the list build keeps lies in neighbouring cells; a dimension with
// fewer than three such cells is not cut (one cell), and the grid is coarsened
// along its longest axis until it has at most kMaxCells cells.
__device__ inline CellGrid cell_grid(const RepConst& c, const double* L) {
  // a cell is wider than any component the FP32 test can keep (its truncated
  // differences err by less than L 2^-16 per component), so the lists equal
  // those of a test against every molecule of the replica
  const double lmax = fmax(fmax(L[0], L[1]), L[2]);
  const double rw = list_test_radius(c, L) + 2.0 * lmax * (1.0 / 65536.0);
  int n[3];
  for (int x = 0; x < 3; x++) {
    const double q = L[x] / rw;
    n[x] = (q >= 3.0) ? (int)fmin(floor(q), (double)kMaxCells) : 1;   // NaN -> 1
  }
  while ((long long)n[0] * n[1] * n[2] > kMaxCells) {
    const int m = (n[0] >= n[1] && n[0] >= n[2]) ? 0 : (n[1] >= n[2] ? 1 : 2);
    n[m] = (n[m] - 1 >= 3) ? n[m] - 1 : 1;
  }
  // A candidate from the cells (gathered, a bitmap bit set) costs several times one of
  // the all-molecule scan (one load tested against four molecules), and the stencil's
  // loops cost a small replica more than its scan.  The lists are the same either way.
  // Lists launches with a quarter of the replicas rebuilt, cut / uncut: 64 tubes of 200
  // molecules (pruned 4x) 23.4 / 14.9 us, of 300 (3x) 24.9 / 20.1, of 450 (6x) 29.2 /
  // 28.4; 16 slits of 1000 (3.6x) 34.9 / 33.4, 8 of 2000 (7x) 34.8 / 51.4, 4 bulk boxes
  // of 4096 (2.4x) 59.5 / 64.7 with 3 us more in the head, of 6000 (4.6x) 111 / 119.
  const int stencil = (n[0] > 1 ? 3 : 1) * (n[1] > 1 ? 3 : 1) * (n[2] > 1 ? 3 : 1);
  if (c.nmol < kCellMinMol || (long long)stencil * kCellMinPrune > (long long)n[0] * n[1] * n[2]) n[0] = n[1] = n[2] = 1;
  CellGrid g;
  g.nx = n[0]; g.ny = n[1]; g.nz = n[2];
  g.rebuild = 1;
  return g;
}

__device__ inline int cell_of(const int4 x, const CellGrid& g) {
  return (cell_coord(x.z, g.nz) * g.ny + cell_coord(x.y, g.ny)) * g.nx + cell_coord(x.x, g.nx);
}

// Per-replica head of a force step, one block per replica of the launch:
//  * warp 0 sums the integrate kernel's partials (lane-strided, then a
//    butterfly, so the order depends only on the replica's record count) and
//    lane 0 runs PsPv and D4 (src/integrator.cxx:132-172, 604-632), writes the
//    replica's scalars to Xout and decides whether its neighbour lists must be
//    rebuilt: pairs now within rc were within rc + skin at the build if
//    2 max|displacement| + rc (max_d Lbuild_d / L_d - 1) <= skin;
//  * when they must, the block counting-sorts the replica's molecules by cell
//    (cell_grid) into cell_start / cell_com; k_force_lists then tests each
//    molecule against the molecules of its 27 (tube: 3, slit: 9) neighbouring
//    cells only.  The order inside a cell is arbitrary: the lists are emitted
//    in ascending j from a bitmap (build_lists), so they do not depend on it.
// This replaces the reference's per-replica z-sort of the molecules
// (sort, src/sort.cu:373-459; quicksort_key, src/quicksort.cu:214-276).
template <bool FORCE_ONLY>
__global__ void __launch_bounds__(kRepThreads) k_replica_head(DevPtrs d, const RepState* __restrict__ Yin,
                                                              RepState* __restrict__ Xout) {
  step_kernel_entry();
  __shared__ int cnt[kMaxCells];
  __shared__ int wsum[kRepThreads / 32];
  __shared__ CellGrid grid;
  const int rep = d.reps ? d.reps[blockIdx.x] : (int)blockIdx.x;
  __shared__ RepConst c;
  __shared__ RepState st0;
  __shared__ double Lb[3];
  {
    const int tid = threadIdx.x;
    const uint32_t* cs = reinterpret_cast<const uint32_t*>(d.rc + rep);
    for (int k = tid; k < (int)(sizeof(RepConst) / 4); k += kRepThreads) reinterpret_cast<uint32_t*>(&c)[k] = cs[k];
    const uint32_t* ys = reinterpret_cast<const uint32_t*>(Yin + rep);
    if (tid >= 64 && tid < 64 + (int)(sizeof(RepState) / 4)) reinterpret_cast<uint32_t*>(&st0)[tid - 64] = ys[tid - 64];
    // every tile of a replica holds the same build box
    if (tid >= 128 && tid < 131) Lb[tid - 128] = d.Lbuild[3 * d.rc[rep].tile_off + tid - 128];
  }
  double v[4] = {0, 0, 0, 0}, disp = 0.0;
  if (!FORCE_ONLY && threadIdx.x < 32) {
    const int w0 = d.rc[rep].warp_off, w1 = w0 + d.rc[rep].nwarp;
    for (int k = w0 + threadIdx.x; k < w1; k += 32) {
      const Part1 p = d.part1[k];
      v[0] += p.sum_Pv[0]; v[1] += p.sum_Pv[1]; v[2] += p.sum_Pv[2];
      v[3] += p.sum_Ps;
      disp = fmax(disp, p.disp);
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double log_s = log(st0.s);   // on every lane, ahead of the sums' exchange
    if (!FORCE_ONLY) {
      warp_sum<4>(v);
      disp = warp_max(disp);
    }
    RepState st = st0;
    int rb = 1;
    if (!FORCE_ONLY) {   // every lane runs the chain (the same bits); lane 0 stores
      pspv(c, st, v, v[3], log_s);
      d4(c, st);
      rb = !(Lb[0] == Lb[0]);
      if (!rb) {
        // lam = max_x Lbuild_x / L_x, one dimension per lane
        const int x = min((int)threadIdx.x, 2);
        double lam = Lb[x] / st.L[x];
        lam = fmax(fmax(__shfl_sync(0xffffffffu, lam, 0), __shfl_sync(0xffffffffu, lam, 1)),
                   __shfl_sync(0xffffffffu, lam, 2));
        rb = (2.0 * disp + c.rc * (lam - 1.0) > c.skin);
      }
    }
    if (threadIdx.x == 0) {
      Xout[rep] = st;   // FORCE_ONLY launches pass Xout == Yin: unchanged there
      CellGrid g;
      g.nx = g.ny = g.nz = 1;
      if (rb) g = cell_grid(c, st.L);
      g.rebuild = rb;
      grid = g;
      d.cgrid[rep] = g;
    }
  }
  __syncthreads();
  if (!grid.rebuild) return;
  const CellGrid g = grid;
  const int ncell = g.nx * g.ny * g.nz;
  if (ncell == 1) return;   // not cut: the list build scans every molecule
  const int tid = threadIdx.x, T = blockDim.x;
  for (int k = tid; k < ncell; k += T) cnt[k] = 0;
  __syncthreads();
  const int4* com = d.com + c.mol_off;
  for (int li = tid; li < c.nmol; li += T) atomicAdd(&cnt[cell_of(com[li], g)], 1);
  __syncthreads();
  // exclusive scan of the counts: a contiguous run of cells per thread
  const int per = (ncell + T - 1) / T;
  const int k0 = min(tid * per, ncell), k1 = min(k0 + per, ncell);
  int run = 0;
  for (int k = k0; k < k1; k++) run += cnt[k];
  int incl = run;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if ((tid & 31) >= o) incl += y;
  }
  if ((tid & 31) == 31) wsum[tid >> 5] = incl;
  __syncthreads();
  int base = incl - run;
  for (int w = 0; w < (tid >> 5); w++) base += wsum[w];
  int* cs = d.cell_start + (long long)rep * (kMaxCells + 1);
  for (int k = k0; k < k1; k++) {
    const int n = cnt[k];
    cnt[k] = base;
    cs[k] = base;
    base += n;
  }
  if (tid == 0) cs[ncell] = c.nmol;
  __syncthreads();
  int4* cm = d.cell_com + c.mol_off;
  for (int li = tid; li < c.nmol; li += T) {
    int4 x = com[li];
    const int pos = atomicAdd(&cnt[cell_of(x, g)], 1);
    x.w = li;
    cm[pos] = x;
  }
}

// Skin-list rebuild, kGroup lanes per molecule: a warp builds the lists of kWarpMol
// consecutive molecules from li0 on, row-major (molecule li's list at d.nbr +
// nbr_off + li * nbr_stride).  The list of molecule i holds, in ascending j, every j
// that passes the list test:
//  * a replica not cut into cells (CellGrid 1 x 1 x 1): every molecule is tested.  A
//    lane loads one candidate and tests it against the warp's molecules, so that one
//    load serves kWarpMol tests and 32 candidates advance per round; a ballot per
//    molecule places the kept ones in ascending j;
//  * a replica cut into cells (k_replica_head): the molecule's kGroup lanes split
//    the molecules of its neighbouring cells (their centres, sorted by cell, carry
//    the local index in .w) and set the molecule's bitmap row with shared-memory
//    atomics (`win` words per row: molecules [32 w0, 32 (w0 + win)) at a time); the
//    row is then emitted in ascending j, lane sub taking words sub, sub + kGroup,
//    ..., placed by a prefix of their popcounts over the group: the same list.
// The skin list only has to contain every pair within rcut + skin (the per-step
// lists then keep exactly the pairs within rcut), so the test, of both forms, is a
// conservative one in FP32 on the top 16 bits of each fixed-point difference
// (converted with the 1.5*2^23 bit trick, on the FMA pipe), against rcut + skin
// widened by the truncation error sqrt(3) L_max 2^-16 and a relative 1e-5.  It may
// keep a few pairs just beyond rcut + skin; the per-step lists, and therefore the
// results, do not change.
__device__ __forceinline__ bool list_test(const int4 me, const int4 cj, float lsc0, float lsc1, float lsc2,
                                          float rl2f) {
  const float fx = (__int_as_float(0x4B400000 + (wrap_diff(me.x, cj.x) >> 16)) - 12582912.f) * lsc0;
  const float fy = (__int_as_float(0x4B400000 + (wrap_diff(me.y, cj.y) >> 16)) - 12582912.f) * lsc1;
  const float fz = (__int_as_float(0x4B400000 + (wrap_diff(me.z, cj.z) >> 16)) - 12582912.f) * lsc2;
  return fx * fx + fy * fy + fz * fz < rl2f;
}

__device__ void build_lists(const DevPtrs& d, const RepConst& c, int rep, int li0, const double* L,
                                uint32_t* bm, int win) {
  const int lane = threadIdx.x & 31, grp = lane / kGroup, sub = lane % kGroup;
  const float lsc0 = (float)(L[0] * (1.0 / 65536.0)), lsc1 = (float)(L[1] * (1.0 / 65536.0)),
              lsc2 = (float)(L[2] * (1.0 / 65536.0));
  const double rw = list_test_radius(c, L);
  const float rl2f = (float)(rw * rw);
  const int4* com = d.com + c.mol_off;
  uint16_t* nb0 = d.nbr + c.nbr_off + (long long)li0 * c.nbr_stride;
  const int nmol = c.nmol, cap = c.nbr_cap;
  const CellGrid g = d.cgrid[rep];
  int cnt = 0;   // entries of molecule li0 + grp
  if (g.nx * g.ny * g.nz == 1) {
    int4 me[kWarpMol];
    int n[kWarpMol];
#pragma unroll
    for (int m = 0; m < kWarpMol; m++) {
      me[m] = com[min(li0 + m, nmol - 1)];
      n[m] = 0;
    }
    const unsigned below = (1u << lane) - 1u;
    for (int base = 0; base < nmol; base += 32) {
      const int j = base + lane;
      const int4 cj = com[min(j, nmol - 1)];
#pragma unroll
      for (int m = 0; m < kWarpMol; m++) {
        const bool in = j < nmol && j != li0 + m &&
                        list_test(me[m], cj, lsc0, lsc1, lsc2, rl2f);
        const unsigned b = __ballot_sync(0xffffffffu, in);
        const int pos = n[m] + __popc(b & below);
        if (in && pos < cap && li0 + m < nmol) nb0[(long long)m * c.nbr_stride + pos] = (uint16_t)j;
        n[m] += __popc(b);
      }
    }
#pragma unroll
    for (int m = 0; m < kWarpMol; m++) cnt = (grp == m) ? n[m] : cnt;
  } else {
    const int li = li0 + grp;
    const bool valid = li < nmol;
    const int4 me = com[min(li, nmol - 1)];
    uint16_t* nb = nb0 + (long long)grp * c.nbr_stride;
    uint32_t* row = bm + (threadIdx.x / kGroup) * (win | 1);   // odd row length: the molecules' words in distinct banks
    const int W = (nmol + 31) >> 5;
    const int cx = cell_coord(me.x, g.nx), cy = cell_coord(me.y, g.ny), cz = cell_coord(me.z, g.nz);
    const int ox = (g.nx == 1) ? 0 : 1, oy = (g.ny == 1) ? 0 : 1, oz = (g.nz == 1) ? 0 : 1;
    const int* cs = d.cell_start + (long long)rep * (kMaxCells + 1);
    const int4* cm = d.cell_com + c.mol_off;
    for (int w0 = 0; w0 < W; w0 += win) {   // uniform over the warp
      const int nw = min(win, W - w0);
      for (int w = sub; w < nw; w += kGroup) row[w] = 0u;
      __syncwarp();
      const int jlo = 32 * w0, jhi = 32 * (w0 + nw);
      if (valid) {
        for (int dz = -oz; dz <= oz; dz++) {
          int zc = cz + dz;
          zc += (zc < 0) ? g.nz : 0;
          zc -= (zc >= g.nz) ? g.nz : 0;
          for (int dy = -oy; dy <= oy; dy++) {
            int yc = cy + dy;
            yc += (yc < 0) ? g.ny : 0;
            yc -= (yc >= g.ny) ? g.ny : 0;
            for (int dx = -ox; dx <= ox; dx++) {
              int xc = cx + dx;
              xc += (xc < 0) ? g.nx : 0;
              xc -= (xc >= g.nx) ? g.nx : 0;
              const int cell = (zc * g.ny + yc) * g.nx + xc;
              const int e = cs[cell + 1];
              for (int k = cs[cell] + sub; k < e; k += kGroup) {
                const int4 cj = cm[k];
                const int j = cj.w;
                if (j < jlo || j >= jhi || j == li) continue;
                if (list_test(me, cj, lsc0, lsc1, lsc2, rl2f))
                  atomicOr(&row[(j - jlo) >> 5], 1u << (j & 31));
              }
            }
          }
        }
      }
      __syncwarp();
      for (int w = 0; w < nw; w += kGroup) {   // uniform over the warp
        const uint32_t word = (w + sub < nw) ? row[w + sub] : 0u;
        const int n = __popc(word);
        int incl = n;   // inclusive prefix of n over the group's lanes
#pragma unroll
        for (int o = 1; o < kGroup; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o, kGroup);
          if (sub >= o) incl += y;
        }
        int pos = cnt + incl - n;
        uint32_t bits = word;
        while (bits) {
          const int j = jlo + 32 * (w + sub) + (__ffs(bits) - 1);
          bits &= bits - 1u;
          if (pos < cap && valid) nb[pos] = (uint16_t)j;
          pos++;
        }
        cnt += __shfl_sync(0xffffffffu, incl, kGroup - 1, kGroup);
      }
      __syncwarp();   // the row is cleared again for the next window
    }
  }
  if (sub == 0 && li0 + grp < nmol) {
    if (cnt > cap) {
      atomicOr(d.err, kErrNbrOverflow);
      atomicMax(&d.status[rep], 8);
      cnt = cap;
    }
    d.nbr_cnt[c.mol_off + li0 + grp] = cnt;
  }
}

// Wall on the oxygen site of a molecule at (r, q): adds the force to f and
// returns the energy (ForceCalculator::Confined, src/force_calculator.cxx:1527-1566;
// slit: src/remdgpu.cu:1708-1720).
__device__ __forceinline__ double wall_site(const DevPtrs& d, const RepConst& c, const double* q, const double* r,
                                            const double* L, double* f) {
  double o[3];
  body_to_space(q, c.body[0], o);
  const double2* fw = reinterpret_cast<const double2*>(d.wall) + c.wall_off;
  const double dr = c.wall_dr;
  if (c.confined == 1) {
    const double x = r[0] * L[0] + o[0] - L[0] * 0.5;
    const double y = r[1] * L[1] + o[1] - L[1] * 0.5;
    const double r01 = sqrt(x * x + y * y);
    int idx = (r01 >= 0.0) ? (int)fmin(r01 / dr, (double)(c.nfwall - 2)) : 0;   // NaN -> 0
    const double2 w0 = fw[idx], w1 = fw[idx + 1];
    const double fr = (w1.x - w0.x) / dr * (r01 - dr * idx) + w0.x;
    f[0] += fr * x;
    f[1] += fr * y;
    return (w1.y - w0.y) / dr * (r01 - dr * idx) + w0.y;
  }
  const double z = r[2] * L[2] + o[2] - 0.5 * L[2];
  const double za = fabs(z);
  const double dir = (za != 0.0) ? z / za : 1.0;
  int idx = (za >= 0.0) ? (int)fmin(za / dr, (double)(c.nfwall - 2)) : 0;       // NaN -> 0
  const double2 w0 = fw[idx], w1 = fw[idx + 1];
  const double fz = (w1.x - w0.x) / dr * (za - dr * idx) + w0.x;
  f[2] += fz * dir;
  return (w1.y - w0.y) / dr * (za - dr * idx) + w0.y;
}

// ------------------------------------------------------------------ FP32 pair step
// The pair step of the FP32 form, in two kernels, kGroup = 8 lanes per molecule
// (four molecules per warp):
//  * k_force_lists writes the molecule's per-step list: the neighbours within rcut,
//    in the (rcut + skin) list's ascending-j order (and the wall term of a confined
//    molecule).  Under the per-site minimum image "far" pairs, whose COM vector
//    keeps every site-pair component clear of +-L/2, fill the list from the front,
//    the others ("near") from the back;
//  * k_force_pairs computes exactly those pairs, lane sub entries sub, sub + 8, ...
//    (first the near, then the far ones), with no cutoff branch.  A lane's sums are
//    FP32 in registers over at most 32 pairs; then the group's lanes are added
//    in FP64 by a fixed exchange tree that leaves three of the molecule's 24 sums
//    with each lane, and finish_group forms force and torque (A2M).
// Which pairs a lane sums, and in what order, depends on the positions only:
// not on the skin list's age, the tile, the batch or the launch.
struct F32Const {
  float Ls[3], Lf[3], hL[3];
  double L[3];
};

// Per-site minimum image (SIMG) flips a site-pair vector by a box length where
// one of its components crosses +-L/2, so the FP32 and FP64 forms must take the
// same image there.  For a site pair with a component within kImageTol of L/2
// (FP32 rounding of the site vector is below ~4e-6 A) the vector is formed anew
// with the FP64 form's arithmetic (pair_loop_f64: COM vector from the FP64 box
// fractions, site offsets R(q) b in FP64, the image decided on their sum).
constexpr float kImageTol = 2e-5f;

__device__ __noinline__ float3 site_vector_exact(const DevPtrs& d, const PairConst& c, const double* L, int li,
                                                 int j, int kk, int l) {
  const int N = d.N, gi = c.mol_off + li, gj = c.mol_off + j;
  double qi[4], qj[4], si[3], sj[3];
  for (int x = 0; x < 4; x++) { qi[x] = d.q[x * N + gi]; qj[x] = d.q[x * N + gj]; }
  body_to_space(qi, c.body[kk], si);
  body_to_space(qj, c.body[l], sj);
  float v[3];
  for (int x = 0; x < 3; x++) {
    double gr = (d.r[x * N + gi] - d.r[x * N + gj]) * L[x];
    if (gr >= 0.5 * L[x]) gr -= L[x];
    if (gr < -0.5 * L[x]) gr += L[x];
    double rv = gr + si[x] - sj[x];
    if (rv >= 0.5 * L[x]) rv -= L[x];
    if (rv < -0.5 * L[x]) rv += L[x];
    v[x] = (float)rv;
  }
  return make_float3(v[0], v[1], v[2]);
}

// Whether the per-site minimum image can change a pair of this box.
__device__ __forceinline__ bool site_image_f32(const PairConst& c, float L0, float L1, float L2) {
  const float reach = 2.f * (c.rc + 2.f * c.reach);
  return L0 < reach || L1 < reach || L2 < reach;
}

// FP32 sums of one lane over its pairs of a segment.
template <int S>
struct F32Sums {
  float fs[S][3], fc[3], fv[3], lj, cl;
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < S; k++) fs[k][0] = fs[k][1] = fs[k][2] = 0.f;
    fc[0] = fc[1] = fc[2] = 0.f;
    fv[0] = fv[1] = fv[2] = 0.f;
    lj = cl = 0.f;
  }
  // the 24 sums by slot: slots 0..4 the sites' forces, 5 the switching correction,
  // 6 the virial, 7 {LJ, Coulomb, -}
  __device__ __forceinline__ float at(int slot, int x) const {
    if (slot < S) return fs[slot][x];
    if (slot == 5) return fc[x];
    if (slot == 6) return fv[x];
    if (slot == 7) return x == 0 ? lj : x == 1 ? cl : 0.f;
    return 0.f;
  }
};

// 2 / sqrt(x): the SFU's reciprocal square root y and one Newton step,
// y (3 - x y^2), without the division by two (~0.5 ulp; three operations).
__device__ __forceinline__ float two_rsqrt(float x) {
  const float y = rsqrtf(x);
  return y * fmaf(-(x * y), y, 3.f);
}

// Site charge in units of the second charged site's (the hydrogens of the water
// models): TIP3P {-2, 1, 1}, TIP4P {1, 1, -2}, TIP5P {1, 1, -1, -1}.  Powers of two, so
// that their products with the unit's square round as the charges' own would.
template <int S>
__device__ __forceinline__ constexpr float charge_ratio(int k) {
  return S == 3 ? (k == 0 ? -2.f : 1.f) : S == 4 ? (k == 3 ? -2.f : 1.f) : (k >= 3 ? -1.f : 1.f);
}

// The lane's n pairs with molecule li: entries row[0], row[+-kGroup], ... (near
// pairs, IMG, are stored backwards).  ci, si: li's fixed-point centre and site
// offsets.  STD: the charges have the ratios of charge_ratio, and the Coulomb terms of
// site kk carry a factor 8 / (q_kk u^2), u the unit charge, that the switch's factor
// takes back once per site.  Other charges enter as their products, each rounded once
// (in units of one of them they could overflow), with the factor 8 alone.
template <int S, int C0, bool STD, bool IMG>
__device__ __forceinline__ void pair_loop_f32(const DevPtrs& d, const PairConst& c, const F32Const& k32, int li,
                                              const int* ci, const float (*si)[3], const uint16_t* row, int n,
                                              F32Sums<S>& a) {
  constexpr int STRIDE = ((3 + 3 * S) + 3) / 4 * 4;
  constexpr int NV = STRIDE / 4;
  const uint4* base = reinterpret_cast<const uint4*>(d.pack) + c.mol_off;
  const int N = d.N;
  const float Ls0 = k32.Ls[0], Ls1 = k32.Ls[1], Ls2 = k32.Ls[2];
  const float rc = c.rc, rs = c.rs, coef = c.coef;
  const float uu = STD ? c.uu : 1.f;
  constexpr int DIR = IMG ? -kGroup : kGroup;
  // the neighbour's record one pair ahead in registers, its index two pairs ahead
  // (2-5 % faster than loading the record at the top of its own iteration)
  int jcur = (n > 0) ? row[0] : 0, jnext = (n > 1) ? row[DIR] : jcur;
  uint4 next[NV];
#pragma unroll
  for (int m = 0; m < NV; m++) next[m] = __ldg(base + (m * N + jcur));
  for (int k = 0; k < n; k++) {
    const int jthis = jcur;
    uint32_t wj[STRIDE];
#pragma unroll
    for (int m = 0; m < NV; m++) {
      wj[4 * m] = next[m].x; wj[4 * m + 1] = next[m].y; wj[4 * m + 2] = next[m].z; wj[4 * m + 3] = next[m].w;
    }
    jcur = jnext;
#pragma unroll
    for (int m = 0; m < NV; m++) next[m] = __ldg(base + (m * N + jcur));
    row += DIR;
    if (k + 2 < n) jnext = row[DIR];
    const float dx = (float)wrap_diff(ci[0], (int)wj[0]) * Ls0;
    const float dy = (float)wrap_diff(ci[1], (int)wj[1]) * Ls1;
    const float dz = (float)wrap_diff(ci[2], (int)wj[2]) * Ls2;
    // vector between site kk of li (already added to d) and site l of j
    auto vec = [&](float ax, float ay, float az, int kk, int l, float& x, float& y, float& z) {
      x = ax - __uint_as_float(wj[3 + 3 * l]);
      y = ay - __uint_as_float(wj[3 + 3 * l + 1]);
      z = az - __uint_as_float(wj[3 + 3 * l + 2]);
      if (IMG) {
        const float hL0 = k32.hL[0], hL1 = k32.hL[1], hL2 = k32.hL[2];
        if (fabsf(fabsf(x) - hL0) < kImageTol || fabsf(fabsf(y) - hL1) < kImageTol ||
            fabsf(fabsf(z) - hL2) < kImageTol) {
          const float3 v = site_vector_exact(d, c, k32.L, li, jthis, kk, l);
          x = v.x; y = v.y; z = v.z;
        } else {
          if (x >= hL0) x -= k32.Lf[0];
          if (x < -hL0) x += k32.Lf[0];
          if (y >= hL1) y -= k32.Lf[1];
          if (y < -hL1) y += k32.Lf[1];
          if (z >= hL2) z -= k32.Lf[2];
          if (z < -hL2) z += k32.Lf[2];
        }
      }
    };
    const float r2 = dx * dx + dy * dy + dz * dz;
    const float rinv = rsqrtf(r2);
    const float r = r2 * rinv;
    float sw = 1.f, dsw = 0.f;
    if (r > rs) {
      const float r01c = r - rc, r01l = r - rs;
      const float cc = coef * r01c * r01c;
      sw = cc * r01c * (10.f * r01l * r01l - 5.f * r01l * r01c + r01c * r01c);
      dsw = cc * 30.f * r01l * r01l;
    }
    const float swu = sw * (0.125f * uu);
    float elj = 0.f, ecl = 0.f;
    float fpx = 0.f, fpy = 0.f, fpz = 0.f;
#pragma unroll
    for (int kk = 0; kk < S; kk++) {
      if (kk != 0 && kk < C0) continue;
      const float ax = dx + si[kk][0], ay = dy + si[kk][1], az = dz + si[kk][2];
      float tx = 0.f, ty = 0.f, tz = 0.f, ek = 0.f;
#pragma unroll
      for (int l = 0; l < S; l++) {
        const bool lj_pair = (kk == 0 && l == 0);
        const bool cl_pair = (kk >= C0 && l >= C0);
        if (!lj_pair && !cl_pair) continue;
        float x, y, z;
        vec(ax, ay, az, kk, l, x, y, z);
        const float ri = two_rsqrt(x * x + y * y + z * z);   // 2 / r
        const float p = ri * ri;                              // 4 / r^2
        if (lj_pair) {
          float s6 = c.sgm2q * p;
          s6 = s6 * s6 * s6;
          const float e4 = c.eps4 * s6;
          elj = e4 * (s6 - 1.f);
          const float f = 3.f * sw * (e4 * (s6 - 0.5f)) * p;
          a.fs[0][0] = fmaf(f, x, a.fs[0][0]);
          a.fs[0][1] = fmaf(f, y, a.fs[0][1]);
          a.fs[0][2] = fmaf(f, z, a.fs[0][2]);
          fpx = f * x; fpy = f * y; fpz = f * z;
        }
        if (cl_pair) {
          const float e = (STD ? charge_ratio<S>(l) : c.qq[kk][l]) * ri;
          ek += e;
          const float f = e * p;
          tx = fmaf(f, x, tx); ty = fmaf(f, y, ty); tz = fmaf(f, z, tz);
        }
      }
      if (kk >= C0) {
        // switch, charge and unit once per site (FFMA into the sums)
        const float qk = STD ? charge_ratio<S>(kk) : 1.f;
        ecl = fmaf(qk, ek, ecl);
        const float w = swu * qk;
        a.fs[kk][0] = fmaf(w, tx, a.fs[kk][0]);
        a.fs[kk][1] = fmaf(w, ty, a.fs[kk][1]);
        a.fs[kk][2] = fmaf(w, tz, a.fs[kk][2]);
        fpx = fmaf(w, tx, fpx); fpy = fmaf(w, ty, fpy); fpz = fmaf(w, tz, fpz);
      }
    }
    ecl *= 0.5f * uu;
    const float g = -(dsw * rinv) * (elj + ecl);
    const float cx = dx * g, cy = dy * g, cz = dz * g;
    a.fc[0] += cx; a.fc[1] += cy; a.fc[2] += cz;
    a.fv[0] = fmaf(fpx + cx, dx, a.fv[0]);
    a.fv[1] = fmaf(fpy + cy, dy, a.fv[1]);
    a.fv[2] = fmaf(fpz + cz, dz, a.fv[2]);
    a.lj = fmaf(sw, elj, a.lj);
    a.cl = fmaf(sw, ecl, a.cl);
  }
}

// Force record of molecule li: its fixed-point centre and site offsets.
template <int S>
__device__ __forceinline__ void load_record(const DevPtrs& d, const PairConst& c, int li, int* ci, float (*si)[3]) {
  constexpr int NV = ((3 + 3 * S) + 3) / 4;
  const uint4* w = reinterpret_cast<const uint4*>(d.pack) + c.mol_off + li;
  uint32_t r[4 * NV];
#pragma unroll
  for (int m = 0; m < NV; m++) {
    const uint4 u = __ldg(w + m * d.N);
    r[4 * m] = u.x; r[4 * m + 1] = u.y; r[4 * m + 2] = u.z; r[4 * m + 3] = u.w;
  }
#pragma unroll
  for (int x = 0; x < 3; x++) ci[x] = (int)r[x];
#pragma unroll
  for (int k = 0; k < S; k++)
#pragma unroll
    for (int x = 0; x < 3; x++) si[k][x] = __uint_as_float(r[3 + 3 * k + x]);
}

// The near pairs of a segment (SIMG), as a call: its image tests and their FP64
// branch would otherwise hold registers through the far pairs' loop (it runs for a few
// percent of the pairs of the boxes close to the minimum-image bound only).  The call
// costs its caller a frame: the kernel that makes it holds the sums whose address it
// takes and spills 144-164 bytes at 128 registers; inlined, it spilled 200.
template <int S, int C0>
__device__ __noinline__ void near_pairs_f32(const DevPtrs& d, const PairConst& c, const F32Const& k32, int li,
                                            const uint16_t* row, int n, F32Sums<S>* out) {
  int ci[3];
  float si[S][3];
  load_record<S>(d, c, li, ci, si);
  F32Sums<S> a;
  a.zero();
  pair_loop_f32<S, C0, false, true>(d, c, k32, li, ci, si, row, n, a);
  *out = a;
}

// One exchange step of the sums' reduction: of 2H values per lane, the lane
// with bit `o` clear keeps the first H and gets its partner's, the other keeps
// the last H; both add the same two numbers.
template <int H>
__device__ __forceinline__ void exchange_sum(double* v, int sub, int o) {
  const bool up = (sub & o) != 0;
#pragma unroll
  for (int k = 0; k < H; k++) {
    const double give = up ? v[k] : v[k + H], keep = up ? v[k + H] : v[k];
    v[k] = keep + __shfl_xor_sync(0xffffffffu, give, o);
  }
}

// Adds the group's eight lanes' sums in FP64: lane sub ends with slot sub.
template <int S>
__device__ __forceinline__ void reduce_sums(const F32Sums<S>& a, int sub, double* acc) {
  double v[12];
  const bool up = (sub & 4) != 0;
#pragma unroll
  for (int k = 0; k < 4; k++)
#pragma unroll
    for (int x = 0; x < 3; x++) {
      // slots k (lower half) and k + 4: exchanged in FP32, added in FP64
      const float lo = a.at(k, x), hi = a.at(k + 4, x);
      const float give = up ? lo : hi, keep = up ? hi : lo;
      v[3 * k + x] = (double)keep + (double)__shfl_xor_sync(0xffffffffu, give, 4);
    }
  exchange_sum<6>(v, sub, 2);
  exchange_sum<3>(v, sub, 1);
#pragma unroll
  for (int x = 0; x < 3; x++) acc[x] += v[x];
}

// Pair forces of molecules li0 .. li0 + kWarpMol - 1 by one warp from their
// per-step lists.  Lane sub of a molecule's group ends with slot sub of its sums in
// acc; returns the molecule's pair count (equal on the group's lanes).
template <int S, int C0, bool STD>
__device__ __forceinline__ int force_warp_f32(const DevPtrs& d, const PairBlk& b, const PairConst& c,
                                              const F32Const& k32, int li0, int nc, double* acc) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, grp = lane / kGroup, sub = lane % kGroup;
  const int lic = min(li0 + grp, b.nmol - 1);
  const int nfar = nc & 0xffff, nnear = nc >> 16;
  const uint16_t* row = d.nbt + b.nbr_off + (long long)lic * b.nbr_stride + sub;
  // FP32 sums close every 32 pairs of a lane: where its near and far pairs together
  // are no more, one segment holds both
  const bool segments = __any_sync(kAll, (nfar + kGroup - 1) / kGroup + (nnear + kGroup - 1) / kGroup >
                                             kSegPairs / kGroup);
  F32Sums<S> a;
  a.zero();
  for (int p0 = 0; __any_sync(kAll, p0 < nnear); p0 += kSegPairs) {
    const int n = min(nnear - p0, kSegPairs) - sub;
    if (n > 0)
      near_pairs_f32<S, C0>(d, c, k32, lic, row + (c.nbr_cap - 1 - p0 - 2 * sub), (n + kGroup - 1) / kGroup, &a);
    if (segments) {
      reduce_sums<S>(a, sub, acc);
      a.zero();
    }
  }
  int ci[3];
  float si[S][3];
  load_record<S>(d, c, lic, ci, si);
  int p0 = 0;
  do {
    const int n = min(nfar - p0, kSegPairs) - sub;
    pair_loop_f32<S, C0, STD, false>(d, c, k32, lic, ci, si, row + p0, (n + kGroup - 1) / kGroup, a);
    __syncwarp();
    reduce_sums<S>(a, sub, acc);
    a.zero();
    p0 += kSegPairs;
  } while (segments && __any_sync(kAll, p0 < nfar));
  return nfar + nnear;
}

// Wall and A2M (FP64) for molecule li of a group of kGroup lanes that hold its
// sums by slot (F32Sums::at), in q4 one component each of q and in wf of the wall
// term {force, energy} (lanes 0..3; both loaded before the pairs): writes d.f and
// d.n, one component per lane.  On return lane 5 of the group holds {wall energy,
// 0, 0}, lane 6 the virial and lane 7 {LJ, Coulomb, pairs} in acc.
template <int S, class Const>
__device__ __forceinline__ void finish_group(const DevPtrs& d, const Const& c, int li, int sub,
                                             double q4, double wf, double* acc, int npairs) {
  const int N = d.N, g = c.mol_off + li;
  const bool valid = li < c.nmol;
  double q[4];
#pragma unroll
  for (int x = 0; x < 4; x++) q[x] = __shfl_sync(0xffffffffu, q4, x, kGroup);
  const double wall_e = __shfl_sync(0xffffffffu, wf, 3, kGroup);
#pragma unroll
  for (int x = 0; x < 3; x++) {
    const double f = __shfl_sync(0xffffffffu, wf, x, kGroup);
    if (sub == 0) acc[x] += f;
  }
  // A2M: molecular force and body torque (src/molecules.cxx:447-475); lane k has
  // site k, lane 5 the switching correction
  double v[8];
  const bool force = sub < S || sub == 5;
#pragma unroll
  for (int x = 0; x < 3; x++) v[x] = force ? acc[x] : 0.0;
  v[3] = v[4] = v[5] = v[6] = v[7] = 0.0;
  if (sub < S) {
    double fb[3];
    space_to_body(q, acc, fb);
    const double* b = c.body[sub];
    v[3] = b[0] * fb[0] + b[1] * fb[1] + b[2] * fb[2];
    v[4] = b[1] * fb[2] - b[2] * fb[1];
    v[5] = b[2] * fb[0] - b[0] * fb[2];
    v[6] = b[0] * fb[1] - b[1] * fb[0];
  }
  exchange_sum<4>(v, sub, 4);
  exchange_sum<2>(v, sub, 2);
  exchange_sum<1>(v, sub, 1);
  if (valid && sub < 3) d.f[sub * N + g] = v[0];
  if (valid && sub >= 3 && sub < 7) d.n[(sub - 3) * N + g] = v[0];
  if (sub == 5) { acc[0] = wall_e; acc[1] = acc[2] = 0.0; }
  if (sub == 7) acc[2] = (double)npairs;
}

// ------------------------------------------------------------------ FP64 form
// One launch per step after the replica head (k_force_f64): per warp of kWarpMol
// molecules, kGroup lanes each, the skin lists where due, then in segments of up to
// kSegPairs pairs per molecule the gather of the neighbours within rcut (tested in
// FP64, ballot-placed in ascending j) into a shared-memory row and the pairs, lane
// sub entries sub, sub + 8, ..., all sums FP64; at the end wall and A2M.  As in the
// FP32 form the pairs a lane sums depend on the positions only.  1/r is one rsqrt
// (its square for 1/r^2) instead of a division and a square root per site pair.
// With one lane per molecule and 128 molecules per block, 800 TIP4P molecules were
// seven blocks, each thread walking a whole list: 224 us a launch, now 22 us (5832
// TIP3P molecules 468 -> 63 us); bound by FP64 latency, and where the grid fills the
// GPU by the FP64 pipe.
template <int S>
struct F64Sums {
  double fs[S][3], fc[3], fv[3], lj, cl;
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < S; k++) fs[k][0] = fs[k][1] = fs[k][2] = 0.0;
    fc[0] = fc[1] = fc[2] = 0.0;
    fv[0] = fv[1] = fv[2] = 0.0;
    lj = cl = 0.0;
  }
  __device__ __forceinline__ double at(int slot, int x) const {   // slots as F32Sums::at
    if (slot < S) return fs[slot][x];
    if (slot == 5) return fc[x];
    if (slot == 6) return fv[x];
    if (slot == 7) return x == 0 ? lj : x == 1 ? cl : 0.0;
    return 0.0;
  }
};

// COM vector of a pair in the minimum image (r: box fractions).
__device__ __forceinline__ void com_vector(const double* ri, const double* rj, const double* L, double* gr) {
#pragma unroll
  for (int x = 0; x < 3; x++) {
    gr[x] = (ri[x] - rj[x]) * L[x];
    if (gr[x] >= 0.5 * L[x]) gr[x] -= L[x];
    if (gr[x] < -0.5 * L[x]) gr[x] += L[x];
  }
}

// SIMG: the minimum image of every site pair, as the reference takes it
// (src/force_calculator.cxx:737-741); it matters only when a box length is below
// 2 (rc + 2 site_reach), and the caller enables it just then.
template <int S, int C0, bool SIMG>
__device__ __forceinline__ void pair_loop_f64(const RepConst& c, const double* pack, const double* L,
                                              const double* wi, const uint16_t* row, int n, F64Sums<S>& a) {
  constexpr int STRIDE = ((3 + 3 * S) + 1) / 2 * 2;
  const double rc = c.rc, rs = c.rs, coef = c.coef_sw;
  for (int k = 0; k < n; k++) {
    const double2* w2 = reinterpret_cast<const double2*>(pack + (long long)row[k * kGroup] * STRIDE);
    double wj[STRIDE];
#pragma unroll
    for (int m = 0; m < STRIDE / 2; m++) {
      const double2 u = __ldg(w2 + m);
      wj[2 * m] = u.x; wj[2 * m + 1] = u.y;
    }
    double gr[3];
    com_vector(wi, wj, L, gr);
    const double r02 = gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2];
    const double rinv = rsqrt(r02);
    const double r = r02 * rinv;
    double sw = 1.0, dsw = 0.0;
    if (r > rs) {
      const double r01c = r - rc, r01l = r - rs, cc = coef * r01c * r01c;
      sw = cc * r01c * (10.0 * r01l * r01l - 5.0 * r01l * r01c + r01c * r01c);
      dsw = cc * 30.0 * r01l * r01l;
    }
    double elj = 0.0, ecl = 0.0, fp[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int kk = 0; kk < S; kk++) {
      if (kk != 0 && kk < C0) continue;
      double t[3] = {0.0, 0.0, 0.0};
#pragma unroll
      for (int l = 0; l < S; l++) {
        const bool lj_pair = (kk == 0 && l == 0);
        const bool cl_pair = (kk >= C0 && l >= C0);
        if (!lj_pair && !cl_pair) continue;
        double v[3];
#pragma unroll
        for (int x = 0; x < 3; x++) {
          v[x] = gr[x] + wi[3 + 3 * kk + x] - wj[3 + 3 * l + x];
          if (SIMG) {
            if (v[x] >= 0.5 * L[x]) v[x] -= L[x];
            if (v[x] < -0.5 * L[x]) v[x] += L[x];
          }
        }
        const double ri = rsqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
        const double ri2 = ri * ri;
        double f = 0.0;
        if (lj_pair) {
          double s6 = c.sgm2 * ri2;
          s6 = s6 * s6 * s6;
          elj = 4.0 * c.eps * s6 * (s6 - 1.0);
          f = 48.0 * c.eps * s6 * (s6 - 0.5) * ri2;
        }
        if (cl_pair) {
          const double e = c.qq[kk][l] * ri;
          ecl += e;
          f += e * ri2;
        }
#pragma unroll
        for (int x = 0; x < 3; x++) t[x] += v[x] * f;
      }
#pragma unroll
      for (int x = 0; x < 3; x++) {
        a.fs[kk][x] += sw * t[x];
        fp[x] += sw * t[x];
      }
    }
    const double g = -(dsw * rinv) * (elj + ecl);
#pragma unroll
    for (int x = 0; x < 3; x++) {
      const double cx = gr[x] * g;
      a.fc[x] += cx;
      a.fv[x] += (fp[x] + cx) * gr[x];
    }
    a.lj += sw * elj;
    a.cl += sw * ecl;
  }
}

// Pair forces of molecules li0 .. li0 + kWarpMol - 1 by one warp, as force_warp_f32;
// `row0` is the warp's buffer.
template <int S, int C0, bool SIMG>
__device__ int force_warp_f64(const DevPtrs& d, const RepConst& c, const double* L, int li0, uint16_t* row0,
                              double* acc) {
  constexpr int STRIDE = ((3 + 3 * S) + 1) / 2 * 2;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, grp = lane / kGroup, sub = lane % kGroup;
  const unsigned group = ((1u << kGroup) - 1u) << (lane - sub), below = group & ((1u << lane) - 1u);
  const int li = li0 + grp, lic = min(li, c.nmol - 1);
  const double* pack = reinterpret_cast<const double*>(d.pack) + c.pack_off;
  const uint16_t* nb = d.nbr + c.nbr_off + (long long)lic * c.nbr_stride;
  const int cnt = (li < c.nmol) ? d.nbr_cnt[c.mol_off + li] : 0;
  double wi[STRIDE];
#pragma unroll
  for (int k = 0; k < STRIDE; k++) wi[k] = pack[(long long)lic * STRIDE + k];
  const double rc2 = c.rc * c.rc;
  auto within = [&](int j) {
    const double* w = pack + (long long)j * STRIDE;
    const double rj[3] = {__ldg(w), __ldg(w + 1), __ldg(w + 2)};
    double gr[3];
    com_vector(wi, rj, L, gr);
    return !(gr[0] * gr[0] + gr[1] * gr[1] + gr[2] * gr[2] > rc2);
  };
  uint16_t* row = row0 + grp * kSegPairs;
  F64Sums<S> a;
  a.zero();
  int pos = 0, skip = 0, npairs = 0;   // list position; pairs of the round at pos already taken
  do {
    int n = 0;
    constexpr int B = 4;   // rounds whose loads are in flight together
    while (true) {
      const bool go = pos < cnt && n < kSegPairs;
      if (!__any_sync(kAll, go)) break;
      if (!__any_sync(kAll, go && (skip > 0 || n + B * kGroup > kSegPairs))) {
        int j[B];
        bool in[B];
#pragma unroll
        for (int m = 0; m < B; m++) {
          const int k = pos + m * kGroup + sub;
          j[m] = (go && k < cnt) ? (int)nb[k] : -1;
        }
#pragma unroll
        for (int m = 0; m < B; m++) in[m] = within(max(j[m], 0)) && j[m] >= 0;
#pragma unroll
        for (int m = 0; m < B; m++) {
          const unsigned b = __ballot_sync(kAll, in[m]);
          if (in[m]) row[n + __popc(b & below)] = (uint16_t)j[m];
          n += __popc(b & group);
        }
        if (go) pos += B * kGroup;
      } else {
        // one round, cut exactly at the segment's last pair
        const int k = pos + sub;
        const int j = (go && k < cnt) ? (int)nb[k] : -1;
        const bool in = j >= 0 && within(j);
        const unsigned b = __ballot_sync(kAll, in);
        const int ord = __popc(b & below) - skip, left = __popc(b & group) - skip;
        const int take = min(left, kSegPairs - n);
        if (in && ord >= 0 && ord < take) row[n + ord] = (uint16_t)j;
        if (go) {
          n += take;
          const bool all = take == left;
          skip = all ? 0 : skip + take;
          pos += all ? kGroup : 0;
        }
      }
    }
    npairs += n;
    __syncwarp();
    pair_loop_f64<S, C0, SIMG>(c, pack, L, wi, row + sub, (n - sub + kGroup - 1) / kGroup, a);
    __syncwarp();   // the row is free again
  } while (__any_sync(kAll, pos < cnt));
  // the group's lanes added by the exchange tree: lane sub ends with slot sub
  double v[24];
#pragma unroll
  for (int s = 0; s < 8; s++)
#pragma unroll
    for (int x = 0; x < 3; x++) v[3 * s + x] = a.at(s, x);
  exchange_sum<12>(v, sub, 4);
  exchange_sum<6>(v, sub, 2);
  exchange_sum<3>(v, sub, 1);
#pragma unroll
  for (int x = 0; x < 3; x++) acc[x] = v[x];
  return npairs;
}

// The block's partial sums from its lanes' {wall}, {virial}, {LJ, Coulomb, pairs}
// (lanes 5, 6, 7 of each group, finish_group).
__device__ __forceinline__ void write_part2(const DevPtrs& d, int record, double* acc, double (*wsum)[8]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int x = 0; x < 3; x++)
    for (int o = kGroup; o < 32; o <<= 1) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], o);
  if (lane == 5) wsum[warp][0] = acc[0];
  if (lane == 6)
    for (int x = 0; x < 3; x++) wsum[warp][1 + x] = acc[x];
  if (lane == 7)
    for (int x = 0; x < 3; x++) wsum[warp][4 + x] = acc[x];
  __syncthreads();
  if (threadIdx.x == 0) {
    double s[7];
    for (int k = 0; k < 7; k++) {
      s[k] = wsum[0][k];
      for (int w = 1; w < kPairWarps; w++) s[k] += wsum[w][k];
    }
    Part2 p;
    p.wall = s[0];
    p.vir[0] = s[1]; p.vir[1] = s[2]; p.vir[2] = s[3];
    p.lj = s[4]; p.clmb = s[5];
    p.npairs = (long long)llrint(s[6]);
    p.pad = 0.0;
    d.part2[record] = p;
  }
}

__device__ inline bool site_image_needed(const RepConst& c, const double* L) {
  const double reach = c.rc + 2.0 * c.site_reach;
  return (L[0] < 2.0 * reach) || (L[1] < 2.0 * reach) || (L[2] < 2.0 * reach);
}

template <int S, int C0>
__device__ void force_block_f64(const DevPtrs& d, const PairBlk& b, const RepConst& c, const double* L,
                                uint16_t* rows, double (*wsum)[8]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % kGroup;
  const int lw = b.li0 + warp * kWarpMol, li = lw + lane / kGroup, g = b.mol_off + min(li, b.nmol - 1);
  double q4 = 0.0, w[4] = {0.0, 0.0, 0.0, 0.0};   // one component of q; wall force and energy
  if (sub < 4 && li < b.nmol) q4 = d.q[sub * d.N + g];
  if (b.confined && sub == 0 && li < b.nmol) {
    double q[4], r[3];
    for (int x = 0; x < 4; x++) q[x] = d.q[x * d.N + g];
    for (int x = 0; x < 3; x++) r[x] = d.r[x * d.N + g];
    w[3] = wall_site(d, c, q, r, L, w);
  }
  double wf = 0.0;
#pragma unroll
  for (int x = 0; x < 4; x++) {
    const double t = __shfl_sync(0xffffffffu, w[x], 0, kGroup);
    if (sub == x) wf = t;
  }
  double acc[3];
  uint16_t* row0 = rows + warp * kWarpMol * kSegPairs;
  const int npairs = site_image_needed(c, L) ? force_warp_f64<S, C0, true>(d, c, L, lw, row0, acc)
                                             : force_warp_f64<S, C0, false>(d, c, L, lw, row0, acc);
  finish_group<S>(d, c, li, sub, q4, wf, acc, npairs);
  write_part2(d, c.part2_off + b.li0 / kPart2Mol, acc, wsum);
}

// S as k_force_pairs.
template <int S>
__global__ void __launch_bounds__(32 * kPairWarps, 2) k_force_f64(DevPtrs d, const RepState* __restrict__ X) {
  step_kernel_entry();
  extern __shared__ uint32_t bm[];
  __shared__ RepConst c;
  __shared__ uint16_t rows[kPairWarps * kWarpMol * kSegPairs];
  __shared__ double wsum[kPairWarps][8];
  const PairBlk b = d.pblk[blockIdx.x];
  const uint32_t* src = reinterpret_cast<const uint32_t*>(d.rc + b.rep);
  for (int k = threadIdx.x; k < (int)(sizeof(RepConst) / 4); k += 32 * kPairWarps)
    reinterpret_cast<uint32_t*>(&c)[k] = src[k];
  const double L[3] = {X[b.rep].L[0], X[b.rep].L[1], X[b.rep].L[2]};
  const int rebuild = d.cgrid[b.rep].rebuild;
  __syncthreads();
  const int li0 = b.li0 + (threadIdx.x >> 5) * kWarpMol;
  if (rebuild) {
    if (li0 < b.nmol) {
      build_lists(d, c, b.rep, li0, L, bm, d.bm_win);
      const int li = li0 + (threadIdx.x & 31) / kGroup;
      if (threadIdx.x % kGroup == 0 && li < b.nmol) d.ref_com[b.mol_off + li] = d.com[b.mol_off + li];
      __syncwarp();   // the lists, written by all lanes, are read below
    }
    if (threadIdx.x < 3 && b.li0 % b.tile == 0) d.Lbuild[3 * (c.tile_off + b.li0 / b.tile) + threadIdx.x] = L[threadIdx.x];
  }
  if (S == 3 || (S == 0 && c.nsite == 3))
    force_block_f64<3, 0>(d, b, c, L, rows, wsum);
  else if (S == 4 || (S == 0 && c.nsite == 4))
    force_block_f64<4, 1>(d, b, c, L, rows, wsum);
  else
    force_block_f64<5, 1>(d, b, c, L, rows, wsum);
}

// A lane's eight skin-list entries from k on, read 16 bytes at a time.  Also past
// the list's end (the array is padded by kListPad entries); the caller masks those.
__device__ __forceinline__ uint4 list_words(const uint16_t* nb, int k) {
  return *reinterpret_cast<const uint4*>(nb + k);
}

// Per-step list of molecule li by its group of kGroup lanes (the FP32 pair step,
// above): 64 skin-list entries at a time, eight consecutive ones per lane (one
// 16-byte load two rounds ahead, then eight centre loads in flight); a prefix over
// the group places the kept ones.  w0, w1: the lane's entries of the first two
// rounds; me: li's centre.
__device__ __forceinline__ void step_list(const DevPtrs& d, const PairBlk& b, const PairConst& c, int li, int cnt,
                                          const int4 me, uint4 w0, uint4 w1, const double* L) {
  constexpr unsigned kAll = 0xffffffffu;
  const int sub = threadIdx.x % kGroup;
  const int lic = min(li, b.nmol - 1);
  const int4* com = d.com + b.mol_off;
  const long long off = b.nbr_off + (long long)lic * b.nbr_stride;
  const uint16_t* nb = d.nbr + off;
  uint16_t* row = d.nbt + off;
  const float L0 = (float)L[0], L1 = (float)L[1], L2 = (float)L[2];
  const float Ls0 = (float)(L[0] * kFixInv), Ls1 = (float)(L[1] * kFixInv), Ls2 = (float)(L[2] * kFixInv);
  const float rc2 = c.rc2;
  const bool simg = site_image_f32(c, L0, L1, L2);
  // far bound: |d_x| below it keeps every site-pair component below L/2 - kImageTol
  const float m = 2.f * c.reach + kImageTol + 1e-3f;
  const float bnd0 = simg ? 0.5f * L0 - m : 1e30f, bnd1 = simg ? 0.5f * L1 - m : 1e30f,
              bnd2 = simg ? 0.5f * L2 - m : 1e30f;
  const int back = c.nbr_cap - 1;
  int nfar = 0, nnear = 0;
  for (int k = 8 * sub; __any_sync(kAll, k - 8 * sub < cnt); k += 8 * kGroup) {
    const uint4 cur = w0;
    w0 = w1;
    if (k + 16 * kGroup < cnt) w1 = list_words(nb, k + 16 * kGroup);
    int j[8];
    int4 u[8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const unsigned w = (e >> 1) == 0 ? cur.x : (e >> 1) == 1 ? cur.y : (e >> 1) == 2 ? cur.z : cur.w;
      j[e] = (k + e < cnt) ? (int)((e & 1) ? (w >> 16) : (w & 0xffffu)) : 0;
      u[e] = __ldg(com + j[e]);
    }
    unsigned in = 0u, nr = 0u;   // within rcut; of these, near
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const float dx = (float)wrap_diff(me.x, u[e].x) * Ls0, dy = (float)wrap_diff(me.y, u[e].y) * Ls1,
                  dz = (float)wrap_diff(me.z, u[e].z) * Ls2;
      if (k + e < cnt && dx * dx + dy * dy + dz * dz <= rc2) in |= 1u << e;
      if (fabsf(dx) >= bnd0 || fabsf(dy) >= bnd1 || fabsf(dz) >= bnd2) nr |= 1u << e;
    }
    nr &= in;
    const unsigned fr = in & ~nr;
    const int n = __popc(fr) | (__popc(nr) << 16);
    int incl = n;   // inclusive prefix over the group's lanes
#pragma unroll
    for (int o = 1; o < kGroup; o <<= 1) {
      const int y = __shfl_up_sync(kAll, incl, o, kGroup);
      if (sub >= o) incl += y;
    }
    const int total = __shfl_sync(kAll, incl, kGroup - 1, kGroup);
    uint16_t* wf = row + nfar + ((incl - n) & 0xffff);
#pragma unroll
    for (int e = 0; e < 8; e++)
      if (fr >> e & 1u) *wf++ = (uint16_t)j[e];
    if (simg) {
      uint16_t* wn = row + back - nnear - ((incl - n) >> 16);
#pragma unroll
      for (int e = 0; e < 8; e++)
        if (nr >> e & 1u) *wn-- = (uint16_t)j[e];
    }
    nfar += total & 0xffff;
    nnear += total >> 16;
  }
  if (sub == 0 && li < b.nmol) d.nt_cnt[b.mol_off + li] = nfar | (nnear << 16);
}

// FP32 form, first launch after the replica head, kPart2Mol molecules per block:
// their wall terms where confined, their skin lists where the replica's are due, and
// their per-step lists.  A kernel of its own, light on registers: its many warps hide
// the gathered loads' latency, which the pair kernel's four per scheduler do not (the
// gather inside the pair kernel took 12 000 of a warp's 43 000 cycles on 256 replicas,
// 111 432 molecules).  It is bound by the latency of its loads, so all that need only
// the block's descriptor are issued together, and the wall's FP64 chain runs under
// them, a molecule per thread of the first warp (one lane in eight of every warp,
// after the lists: 88.6 us there, now 83.4; 256 tubes of 128 .. 420 molecules 41.0 ->
// 36.0).  Two and four lanes per molecule
// measured slower at every length of the lists (158 and 112 us; on the tubes 64 and 45).
__global__ void __launch_bounds__(32 * kPairWarps, 128 / kPart2Mol) k_force_lists(DevPtrs d, const RepState* __restrict__ X) {
  step_kernel_entry();
  extern __shared__ uint32_t bm[];
  __shared__ PairConst c;
  const PairBlk b = d.pblk[blockIdx.x];
  const int li0 = b.li0 + (threadIdx.x >> 5) * kWarpMol;
  const int sub = threadIdx.x % kGroup, li = li0 + (threadIdx.x & 31) / kGroup, lic = min(li, b.nmol - 1);
  const int g = b.mol_off + lic;
  const uint16_t* nb = d.nbr + b.nbr_off + (long long)lic * b.nbr_stride;
  int cnt = (li < b.nmol) ? d.nbr_cnt[g] : 0;
  uint4 w0 = list_words(nb, 8 * sub), w1 = list_words(nb, 8 * sub + 8 * kGroup);
  const int4 me = d.com[g];
  double qr[7];
  const int wli = b.li0 + threadIdx.x, wg = b.mol_off + min(wli, b.nmol - 1);
  const bool wall = b.confined && threadIdx.x < kPart2Mol && wli < b.nmol;
  if (wall) {
    for (int x = 0; x < 4; x++) qr[x] = d.q[x * d.N + wg];
    for (int x = 0; x < 3; x++) qr[4 + x] = d.r[x * d.N + wg];
  }
  const RepState& st = X[b.rep];
  const double L[3] = {st.L[0], st.L[1], st.L[2]};
  const int rebuild = d.cgrid[b.rep].rebuild;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(d.pc + b.rep);
  for (int k = threadIdx.x; k < (int)(sizeof(PairConst) / 4); k += 32 * kPairWarps)
    reinterpret_cast<uint32_t*>(&c)[k] = src[k];
  __syncthreads();
  if (li0 >= b.nmol) return;
  if (wall) {
    double f[3] = {0.0, 0.0, 0.0};
    const double e = wall_site(d, d.rc[b.rep], qr, qr + 4, L, f);
    double2* w = reinterpret_cast<double2*>(d.wallf + 4 * (long long)wg);
    w[0] = make_double2(f[0], f[1]);
    w[1] = make_double2(f[2], e);
  }
  if (rebuild) {
    const RepConst& rc = d.rc[b.rep];
    build_lists(d, rc, b.rep, li0, L, bm, d.bm_win);
    if (sub == 0 && li < b.nmol) d.ref_com[g] = make_int4(me.x, me.y, me.z, 0);
    if (threadIdx.x < 3 && b.li0 % b.tile == 0)
      d.Lbuild[3 * (rc.tile_off + b.li0 / b.tile) + threadIdx.x] = L[threadIdx.x];
    __syncwarp();   // the lists, written by all lanes, are read below
    cnt = (li < b.nmol) ? d.nbr_cnt[g] : 0;
    w0 = list_words(nb, 8 * sub);
    w1 = list_words(nb, 8 * sub + 8 * kGroup);
  }
  step_list(d, b, c, li, cnt, me, w0, w1, L);
}

// FP32 form, second launch of a step: pair forces and A2M of kPart2Mol molecules per
// block, and their partial sums.  Bound by the issue of FP32 instructions at four warps
// per scheduler, then by the latency of a warp's other phases (lists and constants,
// exchange and A2M).  The kernel parameter is a grid constant: near_pairs_f32 takes its
// address, and every thread would copy its 350 bytes into local memory first (256
// replicas, 111 432 molecules: 236 us a launch with that copy, 218 without; 64 tubes of
// 700 TIP4P molecules 58 -> 47, 8 of 4096 48 -> 39, 64 slits of 512 57 -> 51; with two
// threads per molecule instead of eight 272, 54, 55 and 78).  128 registers for all
// models: 168 measured 2-4 % slower, 96 slower still.
template <int S, int C0, bool STD>
__device__ void force_block_f32(const DevPtrs& d, const PairBlk& b, const PairConst& c, const F32Const& k32, int nc,
                                double q4, double wf, double (*wsum)[8]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, sub = lane % kGroup;
  const int lw = b.li0 + warp * kWarpMol;
  double acc[3] = {0.0, 0.0, 0.0};
  const int npairs = force_warp_f32<S, C0, STD>(d, b, c, k32, lw, nc, acc);
  finish_group<S>(d, c, lw + lane / kGroup, sub, q4, wf, acc, npairs);
  write_part2(d, c.part2_off + b.li0 / kPart2Mol, acc, wsum);
}

// S: the sites of every replica of the launch (0: mixed models, chosen per
// block); STD: every replica has the charge ratios of charge_ratio.
template <int S, bool STD>
__global__ void __launch_bounds__(32 * kPairWarps, kPairBlocks) k_force_pairs(const __grid_constant__ DevPtrs d,
                                                                             const RepState* __restrict__ X) {
  step_kernel_entry();
  __shared__ PairConst c;
  __shared__ F32Const k32;
  __shared__ double wsum[kPairWarps][8];
  const PairBlk b = d.pblk[blockIdx.x];
  // loads that need only the block's descriptor
  const int sub = threadIdx.x % kGroup, li = b.li0 + threadIdx.x / kGroup, g = b.mol_off + min(li, b.nmol - 1);
  const int nc = (li < b.nmol) ? d.nt_cnt[g] : 0;
  double q4 = 0.0, wf = 0.0;   // one component each of q and of the wall term
  if (sub < 4 && li < b.nmol) {
    q4 = d.q[sub * d.N + g];
    if (b.confined) wf = d.wallf[4 * (long long)g + sub];
  }
  const uint32_t* src = reinterpret_cast<const uint32_t*>(d.pc + b.rep);
  for (int k = threadIdx.x; k < (int)(sizeof(PairConst) / 4); k += 32 * kPairWarps)
    reinterpret_cast<uint32_t*>(&c)[k] = src[k];
  if (threadIdx.x < 3) {
    const int x = threadIdx.x;
    const double L = X[b.rep].L[x];
    k32.Ls[x] = (float)(L * kFixInv);
    k32.Lf[x] = (float)L;
    k32.hL[x] = 0.5f * (float)L;
    k32.L[x] = L;
  }
  __syncthreads();
  if (S == 3 || (S == 0 && c.nsite == 3))
    force_block_f32<3, 0, STD>(d, b, c, k32, nc, q4, wf, wsum);
  else if (S == 4 || (S == 0 && c.nsite == 4))
    force_block_f32<4, 1, STD>(d, b, c, k32, nc, q4, wf, wsum);
  else
    force_block_f32<5, 1, STD>(d, b, c, k32, nc, q4, wf, wsum);
}

// ------------------------------------------------------------------ per-replica kernels

__device__ inline double barostat_energy(const RepConst& c, const RepState& st) {
  // Molecules::BarostatEnergy (src/molecules.cxx:663-678); slit src/remdgpu.cu:2803-2809
  if (c.pconstant > 0) {
    if (c.confined == 0)
      return 0.5 * (st.Pv[0] * st.Pv[0] + st.Pv[1] * st.Pv[1] + st.Pv[2] * st.Pv[2]) / c.W +
             st.P * st.L[0] * st.L[1] * st.L[2];
    if (c.confined == 1) return 0.5 * st.Pv[2] * st.Pv[2] / c.W + st.P * volume(c, st);
    return (st.Pv[0] * st.Pv[0] + st.Pv[1] * st.Pv[1]) * (0.5 / c.W) + st.P * volume(c, st);
  }
  return 0.0;
}

// Molecules::CalcProperties (src/molecules.cxx:702-734) from the reduced kinetic
// sums; writes the REMDGPU::GetAverages fields (T and pressures reduced).
__device__ inline double calc_properties(const DevPtrs& d, const RepConst& c, const RepState& st,
                                         const double* tra3raw, double rot, double* avg, const P2Sum& e) {
  const double lj = e.lj, clmb = e.clmb, wall = e.wall;
  const double* vir = e.vir;
  const double pot = lj + clmb + wall;
  double tmp[3];
  for (int x = 0; x < 3; x++) {
    const double cf = 1.0 / (st.L[x] * st.s);
    tmp[x] = tra3raw[x] * (cf * cf * 0.5);
  }
  const double tra = tmp[0] + tmp[1] + tmp[2];
  const double kin = tra + rot;
  const double tsm = 0.5 * st.Ps * st.Ps / c.Q;
  const double tsp = st.gkT * log(st.s);
  double tot = pot + kin;
  if (c.tconstant == 1) tot += tsm + tsp;
  if (c.pconstant > 0) tot += barostat_energy(c, st);
  const double V = volume(c, st);
  if (avg) {
    avg[0] = lj; avg[1] = clmb; avg[2] = wall; avg[3] = V;
    avg[4] = tra; avg[5] = rot; avg[6] = kin / (3.0 * c.nmol);
    avg[8] = (tmp[0] * 2.0 + vir[0]) / V;
    avg[9] = (tmp[1] * 2.0 + vir[1]) / V;
    avg[10] = (tmp[2] * 2.0 + vir[2]) / V;
    avg[7] = ((tmp[0] * 2.0 + vir[0]) + (tmp[1] * 2.0 + vir[1]) + (tmp[2] * 2.0 + vir[2])) / (3. * V);
    avg[11] = tot; avg[12] = tot - st.H0;
    avg[13] = st.s; avg[14] = st.Ps;
    avg[15] = st.Pv[0]; avg[16] = st.Pv[1]; avg[17] = st.Pv[2]; avg[18] = 0.0;
  }
  return tot;
}

__device__ inline void kinetic_sums(const DevPtrs& d, const RepConst& c, double s, double* acc) {
  const int N = d.N;
  acc[0] = acc[1] = acc[2] = acc[3] = 0.0;
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    double q[4], p[4];
    for (int x = 0; x < 4; x++) { q[x] = d.q[x * N + g]; p[x] = d.p[x * N + g]; }
    for (int x = 0; x < 3; x++) {
      const double v = d.v[x * N + g];
      acc[x] += (v * v) * c.mass;
    }
    acc[3] += rot_energy(q, p, c.I, s);
  }
}

__device__ inline void finish_replica(const DevPtrs& d, const RepConst& c, int rep, const RepState& st) {
  double* avg = d.avg + (long long)rep * kNumAvg;
  bool ok = true;
  for (int k = 0; k < kNumAvg; k++) ok = ok && isfinite(avg[k]);
  if (!ok) {
    atomicOr(d.err, kErrNonFinite);
    atomicMax(&d.status[rep], 4);
  }
}

__global__ void __launch_bounds__(kRepThreads) k_replica_end(DevPtrs d, RepState* X) {
  __shared__ RepState st;
  __shared__ double cv[4];
  __shared__ double red[8 * 4];
  const int rep = blockIdx.x;
  const RepConst& c = d.rc[rep];
  P2Sum e;
  if (threadIdx.x < 32) e = reduce_part2(d, c.part2_off, c.npart2);
  if (threadIdx.x == 0) {
    RepState s = X[rep];
    for (int x = 0; x < 3; x++) cv[x] = s.L[x] * s.s * c.dthalf * c.im;
    cv[3] = 2.0 * s.s * c.dthalf;
    d5_apply(s, d5_terms(c, s, e.lj + e.clmb + e.wall, e.vir));
    d6(c, s);
    st = s;
  }
  __syncthreads();
  const int N = d.N;
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    double v[3], p[4], q[4], f[3], n[4];
    for (int x = 0; x < 3; x++) { v[x] = d.v[x * N + g]; f[x] = d.f[x * N + g]; }
    for (int x = 0; x < 4; x++) { q[x] = d.q[x * N + g]; p[x] = d.p[x * N + g]; n[x] = d.n[x * N + g]; }
    kick(v, p, q, f, n, cv, cv[3]);
    for (int x = 0; x < 3; x++) d.v[x * N + g] = v[x];
    for (int x = 0; x < 4; x++) d.p[x * N + g] = p[x];
  }
  __syncthreads();
  double acc[4];
  kinetic_sums(d, c, st.s, acc);
  block_sum<4>(acc, red);
  if (threadIdx.x == 0) {
    calc_properties(d, c, st, acc, acc[3], d.avg + (long long)rep * kNumAvg, e);
    X[rep] = st;
    finish_replica(d, c, rep, st);
  }
}

// Initial properties after the first force call: gkT, CalcProperties, H0 = tot
// (Molecules::InitializeProperty, src/molecules.h:260-270).
__global__ void __launch_bounds__(kRepThreads) k_replica_props(DevPtrs d, RepState* X) {
  __shared__ double red[8 * 4];
  const int rep = blockIdx.x;
  const RepConst& c = d.rc[rep];
  RepState st = X[rep];
  double acc[4];
  kinetic_sums(d, c, st.s, acc);
  block_sum<4>(acc, red);
  P2Sum e;
  if (threadIdx.x < 32) e = reduce_part2(d, c.part2_off, c.npart2);
  if (threadIdx.x == 0) {
    st.gkT = 6.0 * (double)c.nmol * st.T;
    double* avg = d.avg + (long long)rep * kNumAvg;
    st.H0 = calc_properties(d, c, st, acc, acc[3], avg, e);
    avg[12] = 0.0;
    X[rep] = st;
  }
}

// Molecules::KillAngularMomentumInTube (src/molecules.cxx:189-210) for the
// replica of this block: the mean angular momentum about the tube axis, taken
// out of molecules further than 1 A from it; L and s from st.
__device__ void kill_tube_angular_block(const DevPtrs& d, const RepConst& c, const RepState& st,
                                        double* red) {
  const int N = d.N;
  double am[4] = {0, 0, 0, 0};
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    double r[3], v[3];
    for (int x = 0; x < 3; x++) {
      r[x] = (d.r[x * N + g] - 0.5) * st.L[x];
      v[x] = d.v[x * N + g] / (st.L[x] * st.s);
    }
    am[0] += c.mass * (r[0] * v[1] - r[1] * v[0]);
    am[1] += c.mass;
  }
  block_sum<4>(am, red);
  const double lz = am[0] / am[1];
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    double r[3];
    for (int x = 0; x < 3; x++) r[x] = (d.r[x * N + g] - 0.5) * st.L[x];
    const double r02 = r[0] * r[0] + r[1] * r[1];
    if (r02 > 1.0) {
      d.v[g] += lz * r[1] / r02 * st.L[0] * st.s;
      d.v[N + g] -= lz * r[0] / r02 * st.L[1] * st.s;
    }
  }
  __syncthreads();
}

// Molecules::KillMomentum (src/molecules.cxx:168-187) for the replica of this
// block: the mean momentum removed along the unconfined directions; in a tube
// (z only) it also removes the angular momentum about the axis.
__device__ void kill_momentum_block(const DevPtrs& d, const RepConst& c, const RepState& st,
                                    double* red) {
  const int N = d.N;
  double acc[4] = {0, 0, 0, 0};
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    for (int x = 0; x < 3; x++) acc[x] += d.v[x * N + g] * c.mass;
    acc[3] += c.mass;
  }
  block_sum<4>(acc, red);
  const double mom[3] = {acc[0] / acc[3], acc[1] / acc[3], acc[2] / acc[3]};
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    if (c.confined == 1) {
      d.v[2 * N + g] -= mom[2];
    } else if (c.confined == 2) {
      d.v[g] -= mom[0];
      d.v[N + g] -= mom[1];
    } else {
      for (int x = 0; x < 3; x++) d.v[x * N + g] -= mom[x];
    }
  }
  __syncthreads();
  if (c.confined == 1) kill_tube_angular_block(d, c, st, red);
}

// The exchange tail for a replica whose condition changed (src/remd.cxx:526-536):
// ChangeTemperature (src/molecules.h:333-353), KillMomentum (+ the tube's angular
// momentum, src/molecules.cxx:168-210), SetPressure, CalcProperties, UpdateHamiltonian.
__global__ void __launch_bounds__(kRepThreads) k_replica_start(DevPtrs d, RepState* X) {
  __shared__ RepState st;
  __shared__ double sh[4];
  __shared__ double red[8 * 4];
  const int rep = blockIdx.x;
  const RepConst& c = d.rc[rep];
  const double Tn = d.newT[rep], Pn = d.newP[rep];
  {
    const RepState s0 = X[rep];
    if (Tn == s0.T && Pn == s0.P) return;   // uniform over the block
  }
  if (threadIdx.x == 0) {
    RepState s = X[rep];
    const double coef = sqrt(Tn / s.T);
    sh[0] = coef / s.s;
    s.Ps *= coef;
    if (c.pconstant == 1) s.Pv[0] *= coef * s.s;
    if (c.pconstant == 2) s.Pv[2] *= coef * s.s;
    if (c.pconstant == 3) { s.Pv[0] *= coef * s.s; s.Pv[1] *= coef * s.s; }
    s.T = Tn;
    s.gkT = 6.0 * (double)c.nmol * s.T;
    s.s = 1.0;
    st = s;
  }
  __syncthreads();
  const int N = d.N;
  const double sc = sh[0];
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    for (int x = 0; x < 3; x++) d.v[x * N + g] *= sc;
    for (int x = 0; x < 4; x++) d.p[x * N + g] *= sc;
  }
  __syncthreads();
  kill_momentum_block(d, c, st, red);
  double kacc[4];
  kinetic_sums(d, c, st.s, kacc);
  block_sum<4>(kacc, red);
  P2Sum e;
  if (threadIdx.x < 32) e = reduce_part2(d, c.part2_off, c.npart2);
  if (threadIdx.x == 0) {
    RepState s = st;
    s.P = Pn;
    s.H0 = calc_properties(d, c, s, kacc, kacc[3], nullptr, e);
    X[rep] = s;
  }
}

// Molecules::VelocityScaling + AngVelocityScaling (src/molecules.cxx:261-311):
// translational and rotational kinetic energies set to 1.5 N T each, momentum
// removed (along z plus the angular momentum about the axis in a tube),
// thermostat and barostat momenta reset.
//  PER_STEP = false: the reference's init_scaling, after which H0 is recomputed
//    (InitializeProperty).  The stored v and p carry a factor s; they are first
//    brought to s = 1 (the reference calls this only at start-up, where s = 1
//    already, and resetting s afterwards would otherwise scale the kinetic
//    energy by 1/s^2).
//  PER_STEP = true: the velocity-scaling thermostat (tconstant 2) before every
//    MD step, for those replicas only, in the reference's exact order (kinetic
//    energy with the current s, then s = 1, then the rotational part); H0 and
//    the averages are left alone.
template <bool PER_STEP>
__global__ void __launch_bounds__(kRepThreads) k_replica_rescale(DevPtrs d, RepState* X) {
  __shared__ RepState st;
  __shared__ double red[8 * 4];
  const int rep = blockIdx.x;
  const RepConst& c = d.rc[rep];
  if (PER_STEP && c.tconstant != 2) return;   // uniform for the block
  if (threadIdx.x == 0) st = X[rep];
  __syncthreads();
  const int N = d.N;
  if (!PER_STEP && st.s != 1.0) {
    const double si = 1.0 / st.s;
    for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
      const int g = c.mol_off + li;
      for (int x = 0; x < 3; x++) d.v[x * N + g] *= si;
      for (int x = 0; x < 4; x++) d.p[x * N + g] *= si;
    }
    __syncthreads();
    if (threadIdx.x == 0) st.s = 1.0;
    __syncthreads();
  }
  double k[4];
  kinetic_sums(d, c, st.s, k);
  block_sum<4>(k, red);
  {
    double tra = 0.0;
    for (int x = 0; x < 3; x++) {
      const double cf = 1.0 / (st.L[x] * st.s);
      tra += k[x] * (cf * cf * 0.5);
    }
    const double coef = (tra > 0.0) ? sqrt(1.5 * c.nmol * st.T / tra) : 1.0;
    for (int li = threadIdx.x; li < c.nmol; li += blockDim.x)
      for (int x = 0; x < 3; x++) d.v[x * N + c.mol_off + li] *= coef;
  }
  __syncthreads();
  kill_momentum_block(d, c, st, red);
  // VelocityScaling takes the tube's angular momentum out once more after KillMomentum
  if (c.confined == 1) kill_tube_angular_block(d, c, st, red);
  __syncthreads();
  if (threadIdx.x == 0) {
    st.s = 1.0;
    st.Ps = 0.0;
    st.Pv[0] = st.Pv[1] = st.Pv[2] = 0.0;
  }
  __syncthreads();
  kinetic_sums(d, c, st.s, k);
  block_sum<4>(k, red);
  {
    const double coef = (k[3] > 0.0) ? sqrt(1.5 * c.nmol * st.T / k[3]) : 1.0;
    for (int li = threadIdx.x; li < c.nmol; li += blockDim.x)
      for (int x = 0; x < 4; x++) d.p[x * N + c.mol_off + li] *= coef;
  }
  __syncthreads();
  if (PER_STEP) {
    if (threadIdx.x == 0) X[rep] = st;
    return;
  }
  kinetic_sums(d, c, st.s, k);
  block_sum<4>(k, red);
  P2Sum e;
  if (threadIdx.x < 32) e = reduce_part2(d, c.part2_off, c.npart2);
  if (threadIdx.x == 0) {
    RepState s = st;
    s.gkT = 6.0 * (double)c.nmol * s.T;
    double* avg = d.avg + (long long)rep * kNumAvg;
    s.H0 = calc_properties(d, c, s, k, k[3], avg, e);
    avg[12] = 0.0;
    X[rep] = s;
  }
}

// ------------------------------------------------------------------ exchange
// Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11): a counter-based generator.
__device__ inline uint4 philox4x32(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
  for (int i = 0; i < 10; i++) {
    const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += W0;
    key.y += W1;
  }
  return ctr;
}

__device__ inline double philox_uniform(unsigned long long seed, long step, int ens, int pair) {
  const uint4 r = philox4x32(make_uint4((uint32_t)pair, (uint32_t)ens, (uint32_t)step,
                                        (uint32_t)((unsigned long long)step >> 32)),
                             make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  const unsigned long long b = ((unsigned long long)r.x << 32 | r.y) >> 11;
  return (double)b * (1.0 / 9007199254740992.0);
}

// REMD::ReplicaExchange + ExchangeList (src/remd.cxx:467-538, src/remdinfo.cxx:54-125),
// one thread per ensemble; pot/vol from the averages of the last interval.
// step < 0: the ensemble's own interval counter (step_ctr[e]) is used and then
// advanced, and the uniforms come from Philox -- the form captured in the
// interval graph.
__global__ void k_exchange(DevPtrs d, const int* grid, const int* rep_off, const int* u_off,
                           int nens, long step_arg, const double* u, const unsigned long long* seeds,
                           int* index, double* T, double* P, long long* step_ctr) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= nens) return;
  long step = step_arg;
  if (step_arg < 0) {
    step = (long)step_ctr[e];
    step_ctr[e] = step + 1;
  }
  const int nt = grid[2 * e], np = grid[2 * e + 1];
  const int off = rep_off[e];
  const int pcon = d.rc[off].pconstant;
  const int ec = (int)(step % 4);
  int* idx = index + off;
  double* Te = T + off;
  double* Pe = P + off;
  auto pot_of = [&](int r) {
    const double* a = d.avg + (long long)(off + r) * kNumAvg;
    return a[0] + a[1] + a[2];
  };
  auto vol_of = [&](int r) { return d.avg[(long long)(off + r) * kNumAvg + 3]; };
  int pair = 0;
  auto trial = [&](int a, int b) {
    const int i1 = idx[a], i2 = idx[b];
    const double b1 = 1. / Te[i1], b2 = 1. / Te[i2];
    double delta = (b2 - b1) * (pot_of(i1) - pot_of(i2));
    if (pcon > 0) delta += (b2 * Pe[i2] - b1 * Pe[i1]) * (vol_of(i1) - vol_of(i2));
    const double uu = u ? u[u_off[e] + pair] : philox_uniform(seeds[e], step, 0, pair);
    pair++;
    if (exp(-delta) > uu) {
      double t = Te[idx[a]]; Te[idx[a]] = Te[idx[b]]; Te[idx[b]] = t;
      t = Pe[idx[a]]; Pe[idx[a]] = Pe[idx[b]]; Pe[idx[b]] = t;
      const int ti = idx[a]; idx[a] = idx[b]; idx[b] = ti;
    }
  };
  if (ec == 0) {
    for (int j = 0; j < np; ++j)
      for (int i = 0; i < nt / 2; ++i) trial(2 * i + j * nt, 2 * i + 1 + j * nt);
  } else if (ec == 1) {
    for (int j = 0; j < np / 2; ++j)
      for (int i = 0; i < nt; ++i) trial(i + 2 * j * nt, i + (2 * j + 1) * nt);
  } else if (ec == 2) {
    for (int j = 0; j < np; ++j)
      for (int i = 0; i < nt / 2 - (nt + 1) % 2; ++i) trial(2 * i + j * nt + 1, 2 * i + 1 + j * nt + 1);
  } else {
    for (int j = 0; j < np / 2 - (np + 1) % 2; ++j)
      for (int i = 0; i < nt; ++i) trial(i + (2 * j + 1) * nt, i + (2 * j + 2) * nt);
  }
}

// ------------------------------------------------------------------ FP32 peak probe
// Eight independent FMA chains per thread, register resident: measures the
// FP32 pipe's FMA throughput (the force kernel's roofline denominator).
__global__ void __launch_bounds__(256) k_fma_peak(float* out, int iters, float a, float b) {
  float x0 = threadIdx.x * 1e-3f, x1 = x0 + 1.f, x2 = x0 + 2.f, x3 = x0 + 3.f;
  float x4 = x0 + 4.f, x5 = x0 + 5.f, x6 = x0 + 6.f, x7 = x0 + 7.f;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int k = 0; k < 16; k++) {
      x0 = fmaf(x0, a, b); x1 = fmaf(x1, a, b); x2 = fmaf(x2, a, b); x3 = fmaf(x3, a, b);
      x4 = fmaf(x4, a, b); x5 = fmaf(x5, a, b); x6 = fmaf(x6, a, b); x7 = fmaf(x7, a, b);
    }
  }
  const float s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (s == 12345.678f) out[blockIdx.x] = s;   // keeps the chains live
}

int measure_fp32_fma(int device, double* ms, long long* flops) {
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return 6;
  const int blocks = prop.multiProcessorCount * 8, threads = 256, iters = 4096;
  float* out = nullptr;
  if (cudaMalloc(&out, blocks * sizeof(float)) != cudaSuccess) return 2;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  k_fma_peak<<<blocks, threads>>>(out, 64, 0.999f, 1e-3f);   // warm-up
  float best = 1e30f;
  for (int rep = 0; rep < 5; rep++) {
    cudaEventRecord(e0);
    k_fma_peak<<<blocks, threads>>>(out, iters, 0.999f, 1e-3f);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    best = fminf(best, t);
  }
  const cudaError_t err = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  if (err != cudaSuccess) return 6;
  *ms = best;
  *flops = (long long)blocks * threads * iters * 16LL * 8LL * 2LL;
  return 0;
}

// Throughput of integer adds into shared memory (64- and 32-bit), into a peer
// block's shared memory (clusters of four) and into global memory (L2): the
// rates at which a pair kernel that computes each pair once could add the
// partner molecule's share of the forces.  Fixed-point sums do not depend on
// the order of their terms, so such a kernel would stay deterministic.  Each
// thread adds to pseudo-random words of a per-block array of kAtomWords words
// (7 values x 736 molecules); every index is taken modulo that size.
constexpr int kAtomWords = 7 * 736;
constexpr int kAtomThreads = 512, kAtomBlocksPerSM = 4, kAtomIters = 4096;

__device__ __forceinline__ unsigned atom_hash(unsigned x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}

template <int MODE>   // 0 shared u64, 1 shared u32, 2 u64 into cluster peers, 3 global u64
__global__ void __launch_bounds__(kAtomThreads) k_atomic_rate(unsigned long long* gbuf, unsigned long long* out,
                                                              int iters) {
  extern __shared__ unsigned long long ash[];
  for (int k = threadIdx.x; k < kAtomWords; k += blockDim.x) ash[k] = 0ull;
  if (MODE == 2) cg::this_cluster().sync(); else __syncthreads();
  unsigned long long* g = gbuf + (size_t)blockIdx.x * kAtomWords;
  unsigned s = atom_hash(threadIdx.x * 7919u + blockIdx.x * 104729u);
  for (int it = 0; it < iters; it++) {
    s = atom_hash(s + (unsigned)it);
    const int idx = (int)(s % (unsigned)kAtomWords);
    if (MODE == 0) atomicAdd(&ash[idx], (unsigned long long)(s & 1023u));
    if (MODE == 1) atomicAdd(reinterpret_cast<unsigned*>(ash) + idx, s & 1023u);
    if (MODE == 2) atomicAdd(cg::this_cluster().map_shared_rank(ash, (int)((s >> 20) & 3u)) + idx,
                             (unsigned long long)(s & 1023u));
    if (MODE == 3) atomicAdd(g + idx, (unsigned long long)(s & 1023u));
  }
  // a cluster's blocks leave only when no peer adds into their memory any more
  if (MODE == 2) cg::this_cluster().sync(); else __syncthreads();
  unsigned long long t = 0ull;
  for (int k = threadIdx.x; k < kAtomWords; k += blockDim.x) t += ash[k];
  if (t == 0x5eedull) atomicAdd(out, t);   // keeps the adds live
}

int measure_atomics(int device, double* rates) {
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return 6;
  const int blocks = prop.multiProcessorCount * kAtomBlocksPerSM;   // 148 SMs: a multiple of 4
  if (blocks % 4) return 6;
  const size_t smem = kAtomWords * sizeof(unsigned long long);
  unsigned long long *g = nullptr, *out = nullptr;
  if (cudaMalloc(&g, (size_t)blocks * smem) != cudaSuccess) return 2;
  if (cudaMalloc(&out, 8) != cudaSuccess) { cudaFree(g); return 2; }
  cudaMemset(g, 0, (size_t)blocks * smem);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  auto launch = [&](int mode, int iters) {
    if (mode == 2) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(blocks);
      cfg.blockDim = dim3(kAtomThreads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = 4;
      at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = 1;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, k_atomic_rate<2>, g, out, iters);
    } else if (mode == 0) {
      k_atomic_rate<0><<<blocks, kAtomThreads, smem>>>(g, out, iters);
    } else if (mode == 1) {
      k_atomic_rate<1><<<blocks, kAtomThreads, smem>>>(g, out, iters);
    } else {
      k_atomic_rate<3><<<blocks, kAtomThreads, smem>>>(g, out, iters);
    }
  };
  for (int mode = 0; mode < 4; mode++) {
    launch(mode, 64);   // warm-up
    float best = 1e30f;
    for (int rep = 0; rep < 3; rep++) {
      cudaEventRecord(e0);
      launch(mode, kAtomIters);
      cudaEventRecord(e1);
      cudaEventSynchronize(e1);
      float t = 0.f;
      cudaEventElapsedTime(&t, e0, e1);
      best = fminf(best, t);
    }
    rates[mode] = (double)blocks * kAtomThreads * kAtomIters / (best * 1e-3) / 1e9;
  }
  const cudaError_t err = cudaGetLastError();
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(g);
  cudaFree(out);
  return err == cudaSuccess ? 0 : 6;
}

// ------------------------------------------------------------------ caller-buffer variant
// Entry and exit kernels of remd_force_snapshot_noalloc (noalloc.cu): the
// caller's AoS positions/quaternions into the scratch SoA arrays and force
// records, and the scratch results back into the caller's AoS outputs.  The
// constants, tiles and box arrive as a kernel parameter; block 0 stores them
// into the scratch for the force kernels that follow on the same stream.
__global__ void k_noalloc_load(DevPtrs d, const NoAllocSetup setup, RepState* __restrict__ X,
                               const double* __restrict__ r_aos, const double* __restrict__ q_aos) {
  const Tile t = setup.tiles[blockIdx.x];
  const RepConst& c = setup.c;
  const int i = threadIdx.x;
  if (i < t.count) {
    const int li = t.start + i;
    const int g = c.mol_off + li;
    double r[3], q[4];
    for (int x = 0; x < 3; x++) r[x] = r_aos[3 * li + x];
    for (int x = 0; x < 4; x++) q[x] = q_aos[4 * li + x];
    for (int x = 0; x < 3; x++) d.r[x * d.N + g] = r[x];
    for (int x = 0; x < 4; x++) d.q[x * d.N + g] = q[x];
    const int fx[3] = {fix_coord(r[0]), fix_coord(r[1]), fix_coord(r[2])};
    write_pack(d, c, kF32, li, r, q, fx);
  }
  if (i == 0) {
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    d.Lbuild[3 * blockIdx.x] = nan;
    if (blockIdx.x == 0) {
      *const_cast<RepConst*>(d.rc) = setup.c;
      *const_cast<PairConst*>(d.pc) = setup.pc;
      for (int k = 0; k < d.ntiles; k++) const_cast<Tile*>(d.tiles)[k] = setup.tiles[k];
      for (int k = 0; k < d.npblk; k++) const_cast<PairBlk*>(d.pblk)[k] = pair_blk(setup.c, 0, k * kPart2Mol, blockDim.x);
      *X = setup.rs;
      *d.err = 0;
      d.status[0] = 0;
    }
  }
}

// out: lj, clmb, wall, vir[3] (halved like ForceCalculator::Switching), the
// number of unordered pairs within rcut, and the error word (0 = ok).
__global__ void k_noalloc_store(DevPtrs d, double* __restrict__ f_aos, double* __restrict__ n_aos,
                                double* __restrict__ out) {
  const RepConst& c = d.rc[0];
  for (int li = threadIdx.x; li < c.nmol; li += blockDim.x) {
    const int g = c.mol_off + li;
    for (int x = 0; x < 3; x++) f_aos[3 * li + x] = d.f[x * d.N + g];
    for (int x = 0; x < 4; x++) n_aos[4 * li + x] = d.n[x * d.N + g];
  }
  P2Sum e;
  if (threadIdx.x < 32) e = reduce_part2(d, c.part2_off, c.npart2);
  if (threadIdx.x == 0) {
    long long np = 0;
    for (int t = c.part2_off; t < c.part2_off + c.npart2; t++) np += d.part2[t].npairs;
    out[0] = e.lj; out[1] = e.clmb; out[2] = e.wall;
    out[3] = e.vir[0]; out[4] = e.vir[1]; out[5] = e.vir[2];
    out[6] = (double)(np / 2);
    out[7] = (double)*d.err;
  }
}

void launch_noalloc_load(const DevPtrs& d, const NoAllocSetup& setup, RepState* X, const double* r_aos,
                         const double* q_aos, int tile, cudaStream_t s) {
  k_noalloc_load<<<d.ntiles, tile, 0, s>>>(d, setup, X, r_aos, q_aos);
}
void launch_noalloc_store(const DevPtrs& d, double* f_aos, double* n_aos, double* out, cudaStream_t s) {
  k_noalloc_store<<<1, 256, 0, s>>>(d, f_aos, n_aos, out);
}

// ------------------------------------------------------------------ state read-back
// The state of replica `rep` (remd_get_state) laid out as its caller wants it --
// r, v (3 per molecule), q, p (4), f (3), n (4), molecule-major -- straight into
// pinned host memory, followed by the replica's scalars and force sums, so that one
// launch and one wait replace a copy per component (22 of them took 330 us).
__global__ void k_gather_state(DevPtrs d, const RepState* __restrict__ X, int rep, double* __restrict__ out) {
  const RepConst& c = d.rc[rep];
  const int n = c.nmol, N = d.N, per = gridDim.x * blockDim.x;
  const double* src[6] = {d.r, d.v, d.q, d.p, d.f, d.n};
  long long off = 0;
  for (int a = 0; a < 6; a++) {
    const int m = (a == 0 || a == 1 || a == 4) ? 3 : 4;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < m * n; k += per)
      out[off + k] = src[a][(long long)(k % m) * N + c.mol_off + k / m];
    off += (long long)m * n;
  }
  if (blockIdx.x == 0 && threadIdx.x < 32) {
    const P2Sum e = reduce_part2(d, c.part2_off, c.npart2);
    if (threadIdx.x == 0) {
      *reinterpret_cast<RepState*>(out + off) = X[rep];
      double* s = out + off + sizeof(RepState) / sizeof(double);
      s[0] = e.lj; s[1] = e.clmb; s[2] = e.wall;
      s[3] = e.vir[0]; s[4] = e.vir[1]; s[5] = e.vir[2];
    }
  }
}

void launch_gather_state(const DevPtrs& d, const RepState* X, int rep, int nmol, double* out, cudaStream_t s) {
  const int blocks = std::max(1, std::min((4 * nmol + 255) / 256, 64));
  k_gather_state<<<blocks, 256, 0, s>>>(d, X, rep, out);
}

// ------------------------------------------------------------------ carrying replicas between handles
// The serving loop's batch changes: replicas that keep running are copied from
// the previous handle's arrays into the new handle's, on the device.
// src[k] = {first molecule of replica k in the old arrays, old replica} or -1.
__global__ void k_carry_molecules(DevPtrs d, const double* __restrict__ r, const double* __restrict__ v,
                                  const double* __restrict__ q, const double* __restrict__ p, int No,
                                  const int2* __restrict__ src) {
  const Tile t = d.tiles[blockIdx.x];
  const int so = src[t.rep].x;
  const int i = threadIdx.x;
  if (so < 0 || i >= t.count) return;
  const int li = t.start + i;
  const int g = d.rc[t.rep].mol_off + li, go = so + li;
  const int N = d.N;
  for (int x = 0; x < 3; x++) {
    d.r[x * N + g] = r[(long long)x * No + go];
    d.v[x * N + g] = v[(long long)x * No + go];
  }
  for (int x = 0; x < 4; x++) {
    d.q[x * N + g] = q[(long long)x * No + go];
    d.p[x * N + g] = p[(long long)x * No + go];
  }
}

// Per replica: the scalars and the pending condition; per ensemble (sens[e] =
// old ensemble or -1): the exchange's slot -> replica index, interval counter
// and seed.
__global__ void k_carry_replicas(int nrep, int nens, RepState* __restrict__ X, const RepState* __restrict__ Xo,
                                 double* __restrict__ T, double* __restrict__ P, const double* __restrict__ To,
                                 const double* __restrict__ Po, const int2* __restrict__ src,
                                 const int* __restrict__ sens, const int* __restrict__ rep_off,
                                 const int* __restrict__ rep_off_o, const int* __restrict__ nrep_e,
                                 int* __restrict__ index, const int* __restrict__ index_o,
                                 long long* __restrict__ step, const long long* __restrict__ step_o,
                                 unsigned long long* __restrict__ seed,
                                 const unsigned long long* __restrict__ seed_o) {
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nrep; k += gridDim.x * blockDim.x) {
    const int so = src[k].y;
    if (so < 0) continue;
    X[k] = Xo[so];
    T[k] = To[so];
    P[k] = Po[so];
  }
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nens; e += gridDim.x * blockDim.x) {
    const int eo = sens[e];
    if (eo < 0) continue;
    for (int c = 0; c < nrep_e[e]; c++) index[rep_off[e] + c] = index_o[rep_off_o[eo] + c];
    step[e] = step_o[eo];
    seed[e] = seed_o[eo];
  }
}

void launch_carry(const DevPtrs& d, const DevPtrs& o, int tile, const int2* src, RepState* X, const RepState* Xo,
                  double* T, double* P, const double* To, const double* Po, int nens, const int* sens,
                  const int* rep_off, const int* rep_off_o, const int* nrep_e, int* index, const int* index_o,
                  long long* step, const long long* step_o, unsigned long long* seed,
                  const unsigned long long* seed_o, bool molecules, cudaStream_t s) {
  if (molecules) k_carry_molecules<<<d.ntiles, tile, 0, s>>>(d, o.r, o.v, o.q, o.p, o.N, src);
  k_carry_replicas<<<(std::max(d.nrep, nens) + 127) / 128, 128, 0, s>>>(
      d.nrep, nens, X, Xo, T, P, To, Po, src, sens, rep_off, rep_off_o, nrep_e, index, index_o, step, step_o,
      seed, seed_o);
}

// ------------------------------------------------------------------ launchers
void launch_pack(const DevPtrs& d, int prec, int tile, cudaStream_t s) {
  k_pack<<<d.ntiles, tile, 0, s>>>(d, prec);
}
int sm_count() {
  static int n[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 1 << 30;
  if (!n[dev]) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev];
}

// A step kernel (it calls step_kernel_entry first).  With `pdl` (DevPtrs::pdl, the
// engine's rule) it is launched with programmatic stream serialisation.
template <typename... KArgs, typename... Args>
static void launch_step_kernel(bool pdl, void (*k)(KArgs...), unsigned grid, unsigned block, size_t smem,
                               cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, args...);
}

void launch_integrate_prec(const DevPtrs& d, const RepState* X, RepState* Y, bool mid, int tile,
                           int prec, cudaStream_t s) {
  // the scalar chain's own warp where the blocks of all the handle's chains, which run
  // side by side, are resident with it: 16 replicas of 128 molecules 1030 us a 50-step
  // interval with it and 1085 without, 8 of 4096 627 a 10-step interval and 648; 96
  // replicas of 729 molecules (2208 tiles) 2584 with it and 2542 without, 256 replicas
  // (111 432 molecules) 3264 and 3194
  const bool chain = (long long)d.ntiles_h * (tile + 32) <= (long long)sm_count() * 3 * 160;
  void (*k)(DevPtrs, const RepState*, RepState*, int) =
      chain ? (mid ? k_integrate<true, true> : k_integrate<false, true>)
            : (mid ? k_integrate<true, false> : k_integrate<false, false>);
  launch_step_kernel(d.pdl, k, d.ntiles, tile + (chain ? 32 : 0), 0, s, d, X, Y, prec);
}
int max_tile(int prec) { return prec == kF32 ? 64 : 128; }

// Bitmap of the list rebuild: one row of (win | 1) words per molecule of a block.
size_t bitmap_smem_bytes(int mols, int win) { return (size_t)mols * (size_t)(win | 1) * sizeof(uint32_t); }

int bitmap_window(int max_nmol) { return std::min((max_nmol + 31) / 32, kBitmapMaxWords); }

// every block's rebuild bitmaps fit the default limit beside the kernels' static arrays
static_assert(kPart2Mol * (kBitmapMaxWords + 1) * 4 <= 8192, "rebuild bitmaps");

// The force launches of one step; e_head / e_lists (may be null) are recorded
// after the head and after the list kernel (profiling: remd_profile_split).
static void launch_force_impl(const DevPtrs& d, const RepState* Yin, RepState* Xout, int prec, bool force_only,
                              cudaStream_t s, cudaEvent_t e_head, cudaEvent_t e_lists) {
  const RepState* Xc = Xout;
  const bool pdl = d.pdl;
  if (force_only) launch_step_kernel(pdl, k_replica_head<true>, d.nrep_l, kRepThreads, 0, s, d, Yin, Xout);
  else launch_step_kernel(pdl, k_replica_head<false>, d.nrep_l, kRepThreads, 0, s, d, Yin, Xout);
  if (e_head) cudaEventRecord(e_head, s);
  if (prec == kF32) {
    launch_step_kernel(pdl, k_force_lists, d.npblk, 32 * kPairWarps, bitmap_smem_bytes(kPart2Mol, d.bm_win), s, d,
                       Xc);
    if (e_lists) cudaEventRecord(e_lists, s);
    void (*pairs)(DevPtrs, const RepState*);
    switch (d.model_l) {
      case 3: pairs = k_force_pairs<3, false>; break;
      case 4: pairs = k_force_pairs<4, false>; break;
      case 5: pairs = k_force_pairs<5, false>; break;
      case 3 + kStdCharges: pairs = k_force_pairs<3, true>; break;
      case 4 + kStdCharges: pairs = k_force_pairs<4, true>; break;
      case 5 + kStdCharges: pairs = k_force_pairs<5, true>; break;
      case kStdCharges: pairs = k_force_pairs<0, true>; break;
      default: pairs = k_force_pairs<0, false>;
    }
    launch_step_kernel(pdl, pairs, d.npblk, 32 * kPairWarps, 0, s, d, Xc);
  } else {
    if (e_lists) cudaEventRecord(e_lists, s);
    const int sites = d.model_l % kStdCharges;
    void (*force)(DevPtrs, const RepState*) =
        sites == 3 ? k_force_f64<3> : sites == 4 ? k_force_f64<4> : sites == 5 ? k_force_f64<5> : k_force_f64<0>;
    launch_step_kernel(pdl, force, d.npblk, 32 * kPairWarps, bitmap_smem_bytes(kPart2Mol, d.bm_win), s, d, Xc);
  }
}

void launch_force(const DevPtrs& d, const RepState* Yin, RepState* Xout, int prec, bool force_only,
                  cudaStream_t s) {
  launch_force_impl(d, Yin, Xout, prec, force_only, s, nullptr, nullptr);
}

void launch_force_timed(const DevPtrs& d, const RepState* Yin, RepState* Xout, int prec, cudaStream_t s,
                        cudaEvent_t e_head, cudaEvent_t e_lists) {
  launch_force_impl(d, Yin, Xout, prec, false, s, e_head, e_lists);
}
void launch_replica_start(const DevPtrs& d, RepState* X, cudaStream_t s) {
  k_replica_start<<<d.nrep, kRepThreads, 0, s>>>(d, X);
}
void launch_replica_end(const DevPtrs& d, RepState* X, cudaStream_t s) {
  k_replica_end<<<d.nrep, kRepThreads, 0, s>>>(d, X);
}
void launch_replica_props(const DevPtrs& d, RepState* X, cudaStream_t s) {
  k_replica_props<<<d.nrep, kRepThreads, 0, s>>>(d, X);
}
void launch_replica_rescale(const DevPtrs& d, RepState* X, bool per_step, cudaStream_t s) {
  if (per_step) k_replica_rescale<true><<<d.nrep, kRepThreads, 0, s>>>(d, X);
  else k_replica_rescale<false><<<d.nrep, kRepThreads, 0, s>>>(d, X);
}
// ------------------------------------------------------------------ histograms
// One thread per condition slot k (slot c of ensemble e).  The sample is the
// Average of the replica at that condition, per molecule (src/remd.cxx:806-811):
// p = (LJ + CLMB + WALL) / nmol, v = VOL / nmol.  Binning, range check and the
// occupied-range bookkeeping follow REMDInfo::IncrementHistogram
// (src/remdinfo.h:299-321) and Histogram::Increment (src/remdinfo.cxx:38-51);
// KeepAverages adds the 19 fields to the bin.  A sample outside
// [min, max) -- or one whose bin rounds up to kHistBins -- is not counted and
// sets kErrHistRange (the reference exits there).  Each slot has one writer,
// so no atomics are needed on the bins.
__global__ void k_histogram(DevPtrs d, const HistEns* __restrict__ he, const int* __restrict__ rep_off,
                            const int* __restrict__ index) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= d.nrep) return;
  const int e = d.rc[k].ens;
  const HistEns H = he[e];
  if (!H.hist) return;
  const int c = k - rep_off[e];
  const int rep = rep_off[e] + index[k];
  const double* a = d.avg + (long long)rep * kNumAvg;
  const double nmol = (double)d.rc[rep].nmol;
  const double pot = (a[0] + a[1] + a[2]) / nmol;
  const double vol = a[3] / nmol;
  bool ok = !(vol < H.vmin || vol >= H.vmax || pot < H.emin || pot >= H.emax);
  const int v = ok ? (int)((vol - H.vmin) / H.dv) : 0;
  const int p = ok ? (int)((pot - H.emin) / H.de) : 0;
  ok = ok && v >= 0 && v < kHistBins && p >= 0 && p < kHistBins;
  if (!ok) {
    atomicOr(d.err, kErrHistRange);
    return;
  }
  int* b = H.bounds + 5 * c;
  if (b[4] == 0) {
    b[0] = b[1] = v;
    b[2] = b[3] = p;
  }
  b[0] = min(b[0], v);
  b[1] = max(b[1], v);
  b[2] = min(b[2], p);
  b[3] = max(b[3], p);
  b[4] += 1;
  const long long bin = ((long long)c * kHistBins + v) * kHistBins + p;
  H.hist[bin] += 1;
  double* s = H.ave + bin * kNumAvg;
  for (int x = 0; x < kNumAvg; x++) s[x] += a[x];
}

void launch_histogram(const DevPtrs& d, const HistEns* he, const int* rep_off, const int* index,
                      cudaStream_t s) {
  k_histogram<<<(d.nrep + 127) / 128, 128, 0, s>>>(d, he, rep_off, index);
}

void launch_exchange_k(const DevPtrs& d, const int* grid, const int* rep_off, const int* u_off,
                       int nens, long step, const double* u, const unsigned long long* seeds,
                       int* index, double* T, double* P, long long* step_ctr, cudaStream_t s) {
  k_exchange<<<(nens + 63) / 64, 64, 0, s>>>(d, grid, rep_off, u_off, nens, step, u, seeds, index, T,
                                             P, step_ctr);
}

}  // namespace remd
