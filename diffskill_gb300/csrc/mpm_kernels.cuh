// Kernels of the differentiable MLS-MPM substep, templated on
//   T  : particle state and grid precision (float or double)
//   TS : precision of F_tmp, the SVD, the von Mises return map, the stress
//        and their adjoints (float, or double for the FP32_SVD64 mode).
//
// Forward  (MPMSimulator.substep, plb/engine/mpm_simulator.py:307-323):
//   k_p2g      compute_F_tmp + svd + p2g      (122-129, 166-225)
//   k_grid_op  grid_op + Primitive.collide    (231-262, primive_base.py:96-120)
//   k_g2p      g2p                            (265-284)
// Adjoint  (MPMSimulator.substep_grad, 325-345), after recomputing the grid:
//   k_g2p_adj      g2p.grad            scatter into the grid-velocity adjoint
//   k_grid_op_adj  grid_op.grad        per node, tool-pose gradients warp-summed, FP64 atomics
//   k_p2g_adj      p2g.grad + svd_grad + compute_F_tmp.grad (gather)
//
// Particle state is component-major: row k of a frame is st[k*ld + p].
//
// Sparse grid: the scratch grids of a substep are stored block-contiguous
// (blocks of 4x4x4 nodes, 64 nodes = 1 KiB in FP32 per block).  Between substeps
// the p2g grid is zero everywhere and no block is flagged.  p2g adds to the grid
// and flags the blocks that particle stencils touch, k_list_blocks turns the flags
// into a device-side list and clears them, grid_op and grid_op.grad run over that
// list with grid-stride loops (no host round trip; capturable in a CUDA graph), and
// the p2g grid's last reader zeroes its listed blocks (grid_op forward, grid_op.grad
// in the adjoint).  So no pass over the particles only marks blocks and none only
// clears the grid.  One substep of 64 scenes (1.1M particles, 32 us of compulsory
// traffic): with the marking in g2p and a compaction that also clears, p2g 82,
// grid_op 14, g2p 48, clear 8 us; now 85, 14, 37 (34 with the gathers by cell) and 7.  Both kernels store the zeros
// last: next to the load of the same node they cost grid_op 12 us and grid_op.grad
// 12 (34 against 22).  Nodes outside the list hold no mass, so grid_op leaves them at
// zero exactly as the dense reference does; g2p and p2g.grad only read nodes inside
// the list.
#pragma once
#include "../../include/mpm_gb300.h"
#include "mpm_math.cuh"
#include "mpm_svd.cuh"
#include "mpm_tools.cuh"

namespace mpm {

// grid node: (mv or v).xyz, m
template <typename T>
struct alignas(4 * sizeof(T)) Node {
  T x, y, z, w;
};

// material constants of the particle math in the precision S, with the
// products that every thread would otherwise form (on the FP64 pipe, in FP64)
template <typename S>
struct MatConsts {
  S dt, p_mass;
  S mu2ks, lamks;  // 2 mu ks, lam ks
  S ysm;           // yield_stress / (2 mu)
};

template <typename T>
struct Consts {
  MatConsts<float> m32;   // of the constants below
  MatConsts<double> m64;  // the same, rounded to T first
  int n_grid;
  int n_scenes;
  int64_t n_particles;
  int64_t ld;
  int64_t G;    // n_grid^3
  int nb;       // blocks per axis (n_grid / 4)
  int64_t NB3;  // blocks per scene
  T dx, inv_dx, dt, p_mass, p_vol;
  T mu, lam, yield_stress;
  T ks;      // -dt * p_vol * 4 * inv_dx^2 (mpm_simulator.py:214)
  T gdt[3];  // dt * gravity * 30 (mpm_simulator.py:235)
  T ground_friction;
  T x_lo, x_hi;  // g2p clamp bounds (mpm_simulator.py:283)
  unsigned int* status;
};

// Threads per CTA of a particle kernel whose arithmetic is in S.  FP32: 128.
// FP64: one warp.  The FP64 pipe is shared by an SM and bounds these kernels,
// so what counts is how evenly the warps spread over the SMs: 10,000 particles
// are 79 CTAs of 128 threads, four warps on each of 79 SMs and none on the other
// 73, but 313 CTAs of one warp, two or three on every SM.
template <typename S>
constexpr int kParticleThreads = sizeof(S) == 8 ? 32 : 128;

// L2 prefetch of the line holding p (no register, no wait)
MPM_DI void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Programmatic dependent launch (griddepcontrol).  A kernel launched with
// programmatic stream serialization may start while the kernel before it in
// the stream is still running: pdl_wait() returns once that kernel has
// completed and its writes are visible (at once after a plain launch), so a
// thread reads nothing that kernel writes, and writes nothing it reads,
// before its pdl_wait().  pdl_trigger() lets the CTAs of the dependent kernel
// launch from then on (they take SMs this kernel's tail leaves idle).
MPM_DI void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
MPM_DI void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// quadratic B-spline stencil (mpm_simulator.py:201-204); base truncates like
// ti.cast(int)
template <typename T>
struct Stencil {
  int base[3];
  T fx[3];
  T w[3][3];  // w[k][d]
};
template <typename T>
MPM_DI bool make_stencil(const Consts<T>& c, const T* x, Stencil<T>& s) {
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    T t = x[d] * c.inv_dx - T(0.5);
    s.base[d] = (int)t;
    T f = x[d] * c.inv_dx - T(s.base[d]);
    s.fx[d] = f;
    s.w[0][d] = T(0.5) * (T(1.5) - f) * (T(1.5) - f);
    s.w[1][d] = T(0.75) - (f - T(1)) * (f - T(1));
    s.w[2][d] = T(0.5) * (f - T(0.5)) * (f - T(0.5));
    ok = ok && (t > T(-1)) && s.base[d] >= 0 && s.base[d] + 2 < c.n_grid;
  }
  return ok;
}
template <typename T>
MPM_DI T dweight(const Stencil<T>& s, int k, int d) {
  T f = s.fx[d];
  return k == 0 ? -(T(1.5) - f) : (k == 1 ? T(-2) * (f - T(1)) : (f - T(0.5)));
}
template <typename T>
MPM_DI void stencil_derivatives(const Stencil<T>& s, T (&dw)[3][3]) {
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int d = 0; d < 3; ++d) dw[k][d] = dweight(s, k, d);
}
template <typename T>
MPM_DI int64_t node_of(const Consts<T>& c, const Stencil<T>& s, int ox, int oy, int oz) {
  return ((int64_t)(s.base[0] + ox) * c.n_grid + (s.base[1] + oy)) * c.n_grid + (s.base[2] + oz);
}

// Offsets, within one scene's block-contiguous grid, of the stencil nodes
// base+o per axis: node (i,j,k) -> ((bi*nb + bj)*nb + bk)*64 + (li*16 + lj*4 + lk)
struct StencilAddr {
  int ax[3], ay[3], az[3];
  MPM_DI int at(int ox, int oy, int oz) const { return ax[ox] + ay[oy] + az[oz]; }
};
template <typename T>
MPM_DI StencilAddr stencil_addr(const Consts<T>& c, const Stencil<T>& s) {
  StencilAddr a;
  const int nb = c.nb;
#pragma unroll
  for (int o = 0; o < 3; ++o) {
    const int i = s.base[0] + o, j = s.base[1] + o, k = s.base[2] + o;
    a.ax[o] = ((i >> 2) * nb * nb << 6) + ((i & 3) << 4);
    a.ay[o] = ((j >> 2) * nb << 6) + ((j & 3) << 2);
    a.az[o] = ((k >> 2) << 6) + (k & 3);
  }
  return a;
}
// grid coordinates of node l (0..63) of global block gb (= scene*NB3 + local block)
template <typename T>
MPM_DI int block_node(const Consts<T>& c, int64_t gb, int l, int* I) {
  const int scene = (int)(gb / c.NB3);
  const int64_t lb = gb - (int64_t)scene * c.NB3;
  const int nb = c.nb;
  I[0] = (int)(lb / ((int64_t)nb * nb)) * 4 + (l >> 4);
  I[1] = (int)((lb / nb) % nb) * 4 + ((l >> 2) & 3);
  I[2] = (int)(lb % nb) * 4 + (l & 3);
  return scene;
}

// Scatter rows of a warp.  Particles of one grid cell scatter into the same 27
// nodes, so a warp sums them before it goes to memory.  The particles were sorted
// by cell some substeps ago; since then some have moved to a neighbouring cell and
// sit between particles of their old one (after 25 substeps a warp of 32 holds 7
// runs of equal cells but 4 different cells, after 50 substeps 14 and 5).  So the
// warp's lanes are put in order again: lane l's row is its place when the lanes
// are grouped by key, groups in the order of their first lanes.  Bit r of `tails`
// is set when row r ends its group, bit r of `emit` when that group is in the grid
// (lanes out of the grid carry unique keys).
struct WarpRows {
  int row;
  unsigned tails, emit;
  bool first;  // this lane is the first of its group
};
MPM_DI WarpRows warp_rows(long long key, bool ok) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const unsigned peers = __match_any_sync(full, key);
  const int size = __popc(peers), first = __ffs(peers) - 1;
  // rows before each lane's group, if the lane is its first: an exclusive scan
  int before = lane == first ? size : 0;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(full, before, d);
    if (lane >= d) before += t;
  }
  const int end = __shfl_sync(full, before, first);  // rows up to and with this lane's group
  WarpRows w;
  w.row = end - size + __popc(peers & below);
  const unsigned last = 1u << (end - 1);
  w.tails = __reduce_or_sync(full, last);
  w.emit = __reduce_or_sync(full, ok ? last : 0u);
  w.first = lane == first;
  return w;
}

// FP32 row scatter.  Every lane writes what its particle contributes to a node,
// wgt(o) (u + G o) and wgt(o), as the 12 values of u and G's columns, the 9
// products wy wz and the 3 wx; then 27 lanes, one per node o, walk the 32 rows: a
// row is three broadcast 16-byte loads, two weights and nine fused multiply-adds
// (three of them packed pairs) in registers, and a group's end is the same row for
// all lanes, so its sum leaves by one 27-lane red.global.add.v4.f32 without
// divergence.  Before, every lane stored its 27 node values one slab of 9 at a
// time and 27 lanes = 9 nodes x 3 row groups read them back, which closed each
// run three times per substep and diverged over the row groups: 2,850 instructions
// per warp in p2g and 2,288 in g2p.grad, now 2,225 and 1,760 (1.1M particles: p2g 128
// to 81 us, g2p.grad 136 to 86).
constexpr int kStagedGroups = 7;
struct RowStage {
  union {
    struct {
      float4 q0[32];  // u.x, u.y, G00, G10
      float4 q1[32];  // G01, G11, G02, G12
      float4 q2[32];  // u.z, G20, G21, G22
      float wyz[32][9];
      float wx[32][4];
    };
    float4 nodes[kStagedGroups][27];  // g2p.grad, before: the nodes that a group gathers
  };
  Node<float>* base[32];  // grid of the row's scene
  int off[32][12];        // ax[3], ay[3], az[3] of the row's stencil
};
// Packed FP32 pairs (add/mul/fma .f32x2): one instruction for two lanes of
// arithmetic, each rounded as the scalar operation would be
MPM_DI unsigned long long f2_bits(float2 a) { return *reinterpret_cast<unsigned long long*>(&a); }
MPM_DI float2 f2_of(unsigned long long b) { return *reinterpret_cast<float2*>(&b); }
MPM_DI float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c)));
  return f2_of(d);
}
// row r of the stage: the lane's particle (u, G row-major)
MPM_DI void row_put(RowStage& sb, int r, const float* u, const float* G, const Stencil<float>& s) {
  sb.q0[r] = make_float4(u[0], u[1], G[0], G[3]);
  sb.q1[r] = make_float4(G[1], G[4], G[2], G[5]);
  sb.q2[r] = make_float4(u[2], G[6], G[7], G[8]);
#pragma unroll
  for (int oy = 0; oy < 3; ++oy)
#pragma unroll
    for (int oz = 0; oz < 3; ++oz) sb.wyz[r][oy * 3 + oz] = s.w[oy][1] * s.w[oz][2];
  *reinterpret_cast<float4*>(sb.wx[r]) = make_float4(s.w[0][0], s.w[1][0], s.w[2][0], 0.f);
}
MPM_DI void row_addresses(RowStage& sb, int r, const StencilAddr& A, Node<float>* grid) {
  sb.base[r] = grid;
  int4* off = reinterpret_cast<int4*>(sb.off[r]);
  off[0] = make_int4(A.ax[0], A.ax[1], A.ax[2], A.ay[0]);
  off[1] = make_int4(A.ay[1], A.ay[2], A.az[0], A.az[1]);
  off[2] = make_int4(A.az[2], 0, 0, 0);
}
// after a __syncwarp() that follows row_put by all lanes.  W: the fourth value of
// a node gets the weights' sum times wm (else 0).
template <bool W>
MPM_DI void row_scatter(const RowStage& sb, unsigned tails, unsigned emit, float wm) {
  const int lane = threadIdx.x & 31;
  const int node = lane < 27 ? lane : 26;  // lanes 27..31 shadow lane 26 and emit nothing
  const int ox = node / 9, j = node - 9 * ox, oy = j / 3, oz = j - 3 * oy;
  const float fx = (float)ox, fy = (float)oy, fz = (float)oz;
  const float2 fx2 = make_float2(fx, fx), fy2 = make_float2(fy, fy), fz2 = make_float2(fz, fz);
  float2 xy = make_float2(0.f, 0.f), zw = xy;
#pragma unroll 4
  for (int r = 0; r < 32; ++r) {
    const float4 q0 = sb.q0[r], q1 = sb.q1[r], q2 = sb.q2[r];
    const float wgt = sb.wx[r][ox] * sb.wyz[r][j];
    const float2 w2 = make_float2(wgt, wgt);
    float2 v = fma2(fx2, make_float2(q0.z, q0.w), make_float2(q0.x, q0.y));
    v = fma2(fy2, make_float2(q1.x, q1.y), v);
    v = fma2(fz2, make_float2(q1.z, q1.w), v);
    const float z = fmaf(fz, q2.w, fmaf(fy, q2.z, fmaf(fx, q2.y, q2.x)));
    xy = fma2(w2, v, xy);
    zw = fma2(w2, make_float2(z, W ? 1.f : 0.f), zw);
    if ((tails >> r) & 1u) {  // the same row for the whole warp
      if (((emit >> r) & 1u) && lane < 27)
        atomicAdd(reinterpret_cast<float4*>(sb.base[r] + (sb.off[r][ox] + sb.off[r][3 + oy] + sb.off[r][6 + oz])),
                  make_float4(xy.x, xy.y, zw.x, W ? wm * zw.y : 0.f));
      xy = zw = make_float2(0.f, 0.f);
    }
  }
}

// FP64 slab scatter.  The 27-node stencil is scattered one ox slab (9 nodes) at a
// time: every lane writes its 9 node values into its row of v and u, then lanes
// 0..26 read the table by columns, lane = g + 3 j summing column j over rows
// [11 g, 11 g + 11).  Each run of equal keys closed inside a row group issues its
// atomics; the run still open at the end of a group is carried into the next by
// two shuffles.  A node's four values are two double2, each in a table of its own
// with row stride 9 x 16 B: stores and loads fall in distinct 16-byte bank groups
// within each quarter warp.  (The FP32 row scatter would take 13 FP64 operations
// per row and lane, 416 per warp, against some 360 here.)  The shuffle scan that
// FP64 took before cost 4 x 5 additions per node and lane; summed by columns it is
// 33 rows x 4 per slab and lane (37,001 particles: p2g 115 -> 68 us, g2p.grad
// 81 -> 59 us).
struct SlabStage {
  double2 v[33][9], u[33][9];  // (x, y) and (z, w); row 32: read, never used
  Node<double>* base[32];      // grid of the row's scene + ax[ox] of the row's base cell
  int ay[32][3], az[32][3];
};
MPM_DI void slab_addresses(SlabStage& sb, int row, const StencilAddr& A) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    sb.ay[row][k] = A.ay[k];
    sb.az[row][k] = A.az[k];
  }
}
// Called between two __syncwarp()s, after all lanes wrote their row of sb.v and
// sb.u.  W: the fourth value is summed too, and multiplied by wm when it is added
// to the grid (p2g: the weights' sum times the particle mass).
template <bool W>
MPM_DI void slab_reduce64(const SlabStage& sb, unsigned tails, unsigned emit, double wm) {
  const int lane = threadIdx.x & 31;
  // lanes 27..31 (g = 3) read lane 24's cells (a broadcast) and emit nothing
  const int g = lane < 27 ? lane % 3 : 3;
  const int j = lane < 27 ? lane / 3 : 8;
  const int oy = j / 3, oz = j - 3 * (j / 3);
  const int r0 = 11 * (g < 3 ? g : 0);
  const unsigned mine = g < 3 ? tails >> r0 : 0u;  // group 2: bit 10 (row 32) is 0
  double acc[4] = {0.0, 0.0, 0.0, 0.0}, head[4] = {0.0, 0.0, 0.0, 0.0};
  int head_row = -1;
  auto put = [&](int r, const double* a) {
    if (!((emit >> r) & 1u)) return;
    Node<double>* n = sb.base[r] + sb.ay[r][oy] + sb.az[r][oz];
    atomicAdd(&n->x, a[0]);
    atomicAdd(&n->y, a[1]);
    atomicAdd(&n->z, a[2]);
    if (W) atomicAdd(&n->w, wm * a[3]);
  };
#pragma unroll 1
  for (int i = 0; i < 11; ++i) {
    const double2 lo = sb.v[r0 + i][j], hi = sb.u[r0 + i][j];
    acc[0] += lo.x;
    acc[1] += lo.y;
    acc[2] += hi.x;
    if (W) acc[3] += hi.y;
    if ((mine >> i) & 1u) {
      if (g > 0 && head_row < 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) head[k] = acc[k];
        head_row = r0 + i;
      } else {
        put(r0 + i, acc);
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = 0.0;
    }
  }
  // acc = the open run at the group's end; group 2 always closes (row 31)
#pragma unroll
  for (int k = 0; k < (W ? 4 : 3); ++k) {
    const double c1 = __shfl_up_sync(0xffffffffu, acc[k], 1);
    const double fwd = acc[k] + ((g == 1 && head_row < 0) ? c1 : 0.0);
    const double c2 = __shfl_up_sync(0xffffffffu, fwd, 1);
    head[k] += g == 1 ? c1 : c2;
  }
  if (g >= 1 && g < 3 && head_row >= 0) put(head_row, head);
}

template <typename T>
struct ScatterStage;
template <>
struct ScatterStage<float> {
  using type = RowStage;
};
template <>
struct ScatterStage<double> {
  using type = SlabStage;
};

template <typename T>
MPM_DI void zero_stencil(Stencil<T>& s) {
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    s.base[d] = 0;
    s.fx[d] = T(1);
#pragma unroll
    for (int k = 0; k < 3; ++k) s.w[k][d] = T(0);
  }
}
template <typename T>
MPM_DI long long cell_key(const Consts<T>& c, int scene, const Stencil<T>& s) {
  return (long long)scene * c.G + ((long long)s.base[0] * c.n_grid + s.base[1]) * c.n_grid + s.base[2];
}

// Loads issued before a kernel's pdl_wait() go to L2 (ld.global.cg): a
// dependent launch may start on an SM whose L1 still holds lines of an older
// content of the same buffer, and only the wait makes the earlier kernels'
// writes visible through L1.  L2 is coherent, and everything these loads read
// was written by kernels that completed before this one started.
template <typename T>
MPM_DI void load_row_cg(const T* __restrict__ st, int64_t ld, int64_t p, int r0, int n, T* out) {
#pragma unroll
  for (int k = 0; k < n; ++k) out[k] = __ldcg(st + (int64_t)(r0 + k) * ld + p);
}
template <typename T>
MPM_DI void load_row(const T* __restrict__ st, int64_t ld, int64_t p, int r0, int n, T* out) {
#pragma unroll
  for (int k = 0; k < n; ++k) out[k] = st[(int64_t)(r0 + k) * ld + p];
}
template <typename T>
MPM_DI void store_row(T* __restrict__ st, int64_t ld, int64_t p, int r0, int n, const T* in) {
#pragma unroll
  for (int k = 0; k < n; ++k) st[(int64_t)(r0 + k) * ld + p] = in[k];
}

// ---------------------------------------------------------------------------
// per-particle p2g math: F_tmp, SVD, von Mises, stress (mpm_simulator.py:
// 122-124, 127-129, 166-182, 205-215) in the precision S
// ---------------------------------------------------------------------------
template <typename S>
struct P2G {
  S U[9], s[3], V[9];
  S is[3];   // 1 / s (0: the SVD was plain, see svd3_left32 and svd3_left64)
  S sm1[3];  // s - 1 (FP32: from the shifted SVD, exact as s -> 1)
  S ehat[3], nrm, inrm, dg, k, e[3];  // inrm = 1 / nrm (FP64 only)
  bool yield;
  S J;
  S em1[3];  // singular values of newF minus 1 (e - 1 when yielding, else s - 1)
};
// FP32 p2g math in terms of the displacement D = F_tmp - I.  The stress
// 2 mu (newF - R) newF^T + lam J (J - 1) I is a difference of numbers near 1
// (newF, R, J) when it is evaluated as written; in FP32 that cancellation
// leaves about 1e-7 / |strain| of relative error in every particle's stress
// (1e-4 at a strain of 1e-3), which then drives the trajectory apart from the
// FP64 one.  Here every small quantity is formed directly: D = G + dt C (I + G)
// with G = F - I (exact for F_ii in [0.5, 2]); the SVD of I + D from the
// shifted matrix (svd3_left32) with s - 1; log(s) = log1p(s - 1); the
// projected singular values e - 1 = expm1(eps'); newF - R = U diag(e - 1) V^T;
// J - 1 = det(I + D) - 1 = tr D + (tr(D)^2 - tr(D^2)) / 2 + det D (elastic) or
// expm1(sum eps) (yield: the von Mises map keeps the volume).  The stored F
// of a yielding particle is formed as I + (D + U diag(e - s) V^T), its
// plastic correction e - s = s expm1(-k eps_hat) taken without cancellation,
// so it carries one FP32 rounding, as an elastic particle's I + D does.
// Mathematically the same function as the reference's (mpm_simulator.py:
// 122-129, 166-225).  The stress takes the SVD basis,
// (newF - R) newF^T = U diag((e - 1) e) U^T; new_F (may be null: the
// adjoint's recompute) receives the updated F.
template <bool WithV>
MPM_DI void p2g_particle_f32(const MatConsts<float>& m, const float* C, const float* F, P2G<float>& P,
                             float* affine, float* new_F) {
  float G[9], CG[9], D[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) G[i] = F[i] - ((i % 4 == 0) ? 1.f : 0.f);
  mm(C, G, CG);
#pragma unroll
  for (int i = 0; i < 9; ++i) D[i] = G[i] + m.dt * (C[i] + CG[i]);
  // J - 1 = det(I + D) - 1 by its invariants
  float Jm1 = D[0] + D[4] + D[8];
  {
    float D2 = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) D2 += D[i * 3 + j] * D[j * 3 + i];
    Jm1 += 0.5f * (Jm1 * Jm1 - D2) + det3(D);
  }
  const bool plain = svd3_left32<WithV>(D, 1.f + Jm1, P.U, P.s, P.sm1, P.is, P.V);
  float eps[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    eps[i] = 0.05f < P.s[i] ? log1p_strain(P.sm1[i]) : logf(0.05f);
  }
  const float esum = eps[0] + eps[1] + eps[2];
  const float mean = third(esum);
#pragma unroll
  for (int i = 0; i < 3; ++i) P.ehat[i] = eps[i] - mean;
  P.nrm = sqrtf(dot3(P.ehat, P.ehat) + 1e-8f);
  P.dg = P.nrm - m.ysm;
  P.yield = P.dg > 0.f;
  float* em1 = P.em1;
  float pc[3];  // e - s, the return map's change of the singular values
  if (P.yield) {
    P.k = fast_div(P.dg, P.nrm);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      em1[i] = expm1_strain(eps[i] - P.k * P.ehat[i]);
      P.e[i] = 1.f + em1[i];
      // both small and accurate to ~1e-7 of themselves: the difference keeps that accuracy
      pc[i] = 0.05f < P.s[i] ? em1[i] - P.sm1[i] : P.e[i] - P.s[i];
    }
  } else {
    P.k = 0.f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      P.e[i] = 1.f;
      em1[i] = P.sm1[i];
      pc[i] = 0.f;
    }
  }
  // the return map keeps the volume, unless a singular value sits at the 0.05
  // floor (then J is the product of the clamped values)
  if (P.yield && !(0.05f < P.s[0] && 0.05f < P.s[1] && 0.05f < P.s[2])) Jm1 = expm1f(esum);
  P.J = 1.f + Jm1;
  // (newF - R) newF^T = U diag(e - 1) V^T V diag(e) U^T = U diag((e - 1) e) U^T
  float h[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) h[i] = m.mu2ks * em1[i] * (1.f + em1[i]);
  const float lj = m.lamks * P.J * Jm1;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) {
      float st = P.U[i * 3] * P.U[j * 3] * h[0] + P.U[i * 3 + 1] * P.U[j * 3 + 1] * h[1] +
                 P.U[i * 3 + 2] * P.U[j * 3 + 2] * h[2];
      if (i == j) st += lj;
      affine[i * 3 + j] = st + m.p_mass * C[i * 3 + j];
      if (j != i) affine[j * 3 + i] = st + m.p_mass * C[j * 3 + i];
    }
  if (new_F) {
    if (P.yield) {
      float UP[9], corr[9];
      if (plain) {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) UP[r * 3 + cc] = P.U[r * 3 + cc] * pc[cc];
        mmT(UP, P.V, corr);
      } else {  // U diag(pc) V^T = W (I + D), W = U diag(pc / s) U^T
        float W[9];
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int cc = 0; cc < 3; ++cc) UP[r * 3 + cc] = P.U[r * 3 + cc] * (pc[cc] * P.is[cc]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = i; j < 3; ++j)
            W[i * 3 + j] = W[j * 3 + i] =
                UP[i * 3] * P.U[j * 3] + UP[i * 3 + 1] * P.U[j * 3 + 1] + UP[i * 3 + 2] * P.U[j * 3 + 2];
        mm(W, D, corr);
#pragma unroll
        for (int i = 0; i < 9; ++i) corr[i] += W[i];
      }
#pragma unroll
      for (int i = 0; i < 9; ++i) new_F[i] = (D[i] + corr[i]) + ((i % 4 == 0) ? 1.f : 0.f);
    } else {
#pragma unroll
      for (int i = 0; i < 9; ++i) new_F[i] = D[i] + ((i % 4 == 0) ? 1.f : 0.f);  // F_tmp
    }
  }
}
// FP64 p2g math (mpm_simulator.py:122-129, 166-225) from the left SVD of
// F_tmp (svd3_left64): (newF - R) newF^T = U diag((e - 1) e) U^T, and the
// yielding newF = U diag(e) V^T = F_tmp + U diag(e / s - 1) U^T F_tmp, so the
// forward pass needs no V.  The adjoint's recompute (WithV, new_F null) does.
template <bool WithV>
MPM_DI void p2g_particle_f64(const MatConsts<double>& m, const double* C, const double* F, P2G<double>& P,
                             double* affine, double* new_F) {
  double IC[9], Ftmp[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) IC[i] = m.dt * C[i] + ((i % 4 == 0) ? 1.0 : 0.0);
  mm(IC, F, Ftmp);
  const bool plain = svd3_left64<WithV>(Ftmp, P.U, P.s, P.is, P.V);
  double eps[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    P.sm1[i] = P.s[i] - 1.0;
    eps[i] = 0.05 < P.s[i] ? log_strain64(P.s[i], P.sm1[i]) : log(0.05);
  }
  const double mean = third(eps[0] + eps[1] + eps[2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) P.ehat[i] = eps[i] - mean;
  const double n2 = dot3(P.ehat, P.ehat) + 1e-8;
  P.inrm = rsqrt64_mid(n2);  // (a sum of squared logarithms)
  P.nrm = n2 * P.inrm;
  P.dg = P.nrm - m.ysm;
  P.yield = P.dg > 0.0;
  P.k = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    P.em1[i] = P.sm1[i];
    P.e[i] = P.s[i];
  }
  if (P.yield) {
    P.k = P.dg * P.inrm;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      P.em1[i] = expm1_strain64(fma(-P.k, P.ehat[i], eps[i]));
      P.e[i] = 1.0 + P.em1[i];
    }
  }
  P.J = P.e[0] * P.e[1] * P.e[2];
  double h[3], UH[9];
#pragma unroll
  for (int i = 0; i < 3; ++i) h[i] = m.mu2ks * P.em1[i] * P.e[i];
#pragma unroll
  for (int r = 0; r < 3; ++r)
#pragma unroll
    for (int i = 0; i < 3; ++i) UH[r * 3 + i] = P.U[r * 3 + i] * h[i];
  const double lj = m.lamks * P.J * (P.J - 1.0);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i; j < 3; ++j) {
      double st = UH[i * 3] * P.U[j * 3] + UH[i * 3 + 1] * P.U[j * 3 + 1] + UH[i * 3 + 2] * P.U[j * 3 + 2];
      if (i == j) st += lj;
      affine[i * 3 + j] = st + m.p_mass * C[i * 3 + j];
      if (j != i) affine[j * 3 + i] = st + m.p_mass * C[j * 3 + i];
    }
  if (new_F) {
#pragma unroll
    for (int i = 0; i < 9; ++i) new_F[i] = Ftmp[i];
    if (P.yield) {
      double UW[9];
      if (plain) {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int i = 0; i < 3; ++i) UW[r * 3 + i] = P.U[r * 3 + i] * P.e[i];
        mmT(UW, P.V, new_F);
      } else {
        double W[9];  // U diag(e / s - 1) U^T, symmetric
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int i = 0; i < 3; ++i) UW[r * 3 + i] = P.U[r * 3 + i] * fma(P.e[i], P.is[i], -1.0);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = i; j < 3; ++j)
            W[i * 3 + j] = W[j * 3 + i] =
                UW[i * 3] * P.U[j * 3] + UW[i * 3 + 1] * P.U[j * 3 + 1] + UW[i * 3 + 2] * P.U[j * 3 + 2];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j)
            new_F[i * 3 + j] += W[i * 3] * Ftmp[j] + W[i * 3 + 1] * Ftmp[3 + j] + W[i * 3 + 2] * Ftmp[6 + j];
      }
    }
  }
}
// affine (the APIC matrix with the stress) and, when new_F is given, the
// updated F; P keeps what the adjoint needs (WithV: the adjoint's recompute)
template <bool WithV, typename S>
MPM_DI void p2g_particle(const MatConsts<S>& m, const S* C, const S* F, P2G<S>& P, S* affine, S* new_F) {
  if constexpr (sizeof(S) == 4)
    p2g_particle_f32<WithV>(m, C, F, P, affine, new_F);
  else
    p2g_particle_f64<WithV>(m, C, F, P, affine, new_F);
}
// gradient of the singular values through the return map (yield branch of
// compute_von_mises, mpm_simulator.py:166-180), from the diagonal of
// M_N = U^T g_newF V (d loss / d e_i = M_N,ii)
template <typename S>
MPM_DI void return_map_sigma_grad(const P2G<S>& P, const S* MN, S* gs) {
  S g_eps2[3], g_eps[3], g_ehat[3], g_k = S(0);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    g_eps2[i] = MN[i * 4] * P.e[i];
    g_eps[i] = g_eps2[i];
    g_k -= g_eps2[i] * P.ehat[i];
    g_ehat[i] = -P.k * g_eps2[i];
  }
  S g_nrm;
  if constexpr (sizeof(S) == 8) {
    g_nrm = g_k * P.inrm * (S(1) - P.k);  // k = dg / nrm
#pragma unroll
    for (int i = 0; i < 3; ++i) g_ehat[i] += g_nrm * P.ehat[i] * P.inrm;
  } else {
    g_nrm = -fast_div(g_k * P.dg, P.nrm * P.nrm) + fast_div(g_k, P.nrm);
#pragma unroll
    for (int i = 0; i < 3; ++i) g_ehat[i] += fast_div(g_nrm * P.ehat[i], P.nrm);
  }
  S sh = third(g_ehat[0] + g_ehat[1] + g_ehat[2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    g_eps[i] += g_ehat[i] - sh;
    if constexpr (sizeof(S) == 8)
      gs[i] = (S(0.05) < P.s[i]) ? g_eps[i] * P.is[i] : S(0);
    else
      gs[i] = (S(0.05) < P.s[i]) ? fast_div(g_eps[i], P.s[i]) : S(0);
  }
}

// Adjoint of p2g_particle in the SVD basis.  With G = U^T g_raw U
// (g_raw = ks g_affine), e' = 1 + em1 the singular values of newF, and the
// stress's matrices written in the bases U, V:
//   U^T (g_raw newF) V   = G diag(e')        (the adjoint of A = newF - R)
//   U^T (g_raw^T A) V    = G^T diag(e' - 1)  (through the right factor newF^T)
//   U^T cof(newF) V      = J diag(1 / e')    (d det / d newF; det_grad)
// M_R = U^T g_R V = -2 mu G diag(e') and M_N = U^T g_newF V need no newF, A
// or cofactor matrix.  The SVD part is svd3_bwd_factored_basis; the elastic
// branch's direct newF = F_tmp term joins it in the same basis, so one
// transform U Y V^T gives the gradient of F_tmp.
// g d det(newF) / d e'_i
MPM_DI float det_grad(const P2G<float>& P, float g, int i) { return fast_div(g * P.J, 1.f + P.em1[i]); }
MPM_DI double det_grad(const P2G<double>& P, double g, int i) { return g * (P.e[(i + 1) % 3] * P.e[(i + 2) % 3]); }
template <typename S>
MPM_DI void p2g_particle_vjp(const MatConsts<S>& m, const S* C, const S* F, const P2G<S>& P, const S* g_affine,
                             const S* g_newF_in, S* g_C, S* g_F) {
  S G[9], t9[9], MR[9], MN[9];  // here G = U^T g_affine U: ks is in the constants
  mTm(P.U, g_affine, t9);
  mm(t9, P.U, G);
  const S g_J = m.lamks * (S(2) * P.J - S(1)) * (G[0] + G[4] + G[8]);  // tr g_affine = tr G
  mTm(P.U, g_newF_in, t9);
  mm(t9, P.V, MN);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const S cm = m.mu2ks * P.em1[j], ce = m.mu2ks + cm;  // times e' - 1 and e'
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const S a = ce * G[i * 3 + j];
      MR[i * 3 + j] = -a;
      MN[i * 3 + j] += a + cm * G[j * 3 + i] + (i == j ? det_grad(P, g_J, i) : S(0));
    }
  }
  S gs[3] = {S(0), S(0), S(0)}, Y[9];
  if (P.yield) return_map_sigma_grad(P, MN, gs);
  svd3_bwd_factored_basis(P.s, P.is, P.sm1, MR, MN, P.e, P.em1, S(1) - P.k, P.yield, gs, Y);
  if (!P.yield) {
#pragma unroll
    for (int i = 0; i < 9; ++i) Y[i] += MN[i];  // newF = F_tmp
  }
  S g_Ftmp[9];
  mm(P.U, Y, t9);
  mmT(t9, P.V, g_Ftmp);
  mmT(g_Ftmp, F, t9);  // Ftmp = (I + dt C) F
#pragma unroll
  for (int i = 0; i < 9; ++i) g_C[i] = m.p_mass * g_affine[i] + m.dt * t9[i];
  S IC[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) IC[i] = m.dt * C[i] + ((i % 4 == 0) ? S(1) : S(0));
  mTm(IC, g_Ftmp, g_F);
}

template <typename T, typename S>
MPM_DI const MatConsts<S>& mat_consts(const Consts<T>& c) {
  if constexpr (sizeof(S) == 8)
    return c.m64;
  else
    return c.m32;
}

// flags[scene*NB3 + block] = 1 for the 1, 2, 4 or 8 blocks of the stencil at base, by
// one lane per group of equal cells (`mine`).  Plain byte stores: reading the flags
// and appending the fresh blocks to the list from here made p2g 20 us slower (1.1M
// particles, 102 against 85 us for the stores and 6 for k_list_blocks).
template <typename T>
MPM_DI void flag_blocks(const Consts<T>& c, bool mine, const int* base, int scene, unsigned char* __restrict__ flags) {
  if (!mine) return;
  int lo[3], ext[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d] = base[d] >> 2;
    ext[d] = ((base[d] + 2) >> 2) - lo[d];  // 0 or 1
  }
  const int nb = c.nb;
  unsigned char* f = flags + (int64_t)scene * c.NB3 + ((lo[0] * nb + lo[1]) * nb + lo[2]);
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    const int di = m >> 2, dj = (m >> 1) & 1, dk = m & 1;
    if (di <= ext[0] && dj <= ext[1] && dk <= ext[2]) f[(di * nb + dj) * nb + dk] = 1;
  }
}

// ---------------------------------------------------------------------------
// forward kernels
// ---------------------------------------------------------------------------
struct PoseTableArgs {
  int n_tools;
  const double *pose_f, *pose_f1;
  void* poses;  // T[n_tools * 16]
};
template <typename T>
MPM_DI void pose_table_fill(const PoseTableArgs& a, int64_t i, int64_t stride) {
  for (int64_t j = i; j < (int64_t)a.n_tools * 16; j += stride) {
    const int64_t t = j >> 4;
    const int k = (int)(j & 15);
    static_cast<T*>(a.poses)[j] = T(k < 8 ? a.pose_f[8 * t + k] : a.pose_f1[8 * t + k - 8]);
  }
}
// The particle of thread i of a scattering kernel.  order (may be null): a
// permutation that sorts the particles by cell, for frames that are kept in the
// caller's order; its load before a pdl_wait() goes to L2 (load_row_cg).  The rows
// are then read one sector per particle, which g2p and p2g.grad, with nothing to
// scatter, would only lose by (30,000 particles: g2p 8.8 -> 11.5 us, p2g.grad
// 13.6 -> 35; p2g 24 -> 14, g2p.grad 25 -> 20).
MPM_DI int64_t particle_of(const int* __restrict__ order, int64_t i, bool valid) {
  return order && valid ? (int64_t)__ldcg(order + i) : i;
}
// one chunk of p2g, a particle per thread (all threads of the block take part)
template <typename T, typename S>
MPM_DI void p2g_chunk(const Consts<T>& c, const T* __restrict__ st, T* __restrict__ st_out,
                      const int* __restrict__ pscene, const int* __restrict__ order, Node<T>* __restrict__ grid,
                      unsigned char* __restrict__ flags, int64_t i) {
  const bool valid = i < c.n_particles;  // every lane stays for the warp's scatter
  const int64_t p = particle_of(order, i, valid);
  Stencil<T> s;
  zero_stencil(s);
  bool ok = false;
  int scene = 0;
  // node value of stencil offset o: wgt(o) * (pm + affine o), where
  // affine = dx A and pm = m v - affine fx (= m v + A dp at o = 0, dp = (o - fx) dx);
  // stepped across the stencil by additions of affine's columns
  T affine[9], pm[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int k = 0; k < 9; ++k) affine[k] = T(0);
  if (valid) {
    T x[3], v[3];
    S C[9], F[9];
    load_row_cg(st, c.ld, p, 0, 3, x);
    load_row_cg(st, c.ld, p, 3, 3, v);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      C[k] = to_prec<S>(__ldcg(st + (int64_t)(6 + k) * c.ld + p));
      F[k] = to_prec<S>(__ldcg(st + (int64_t)(15 + k) * c.ld + p));
    }
    const int sc = __ldcg(pscene + p);  // issued with the state rows
    ok = make_stencil(c, x, s);
    const MatConsts<S>& m = mat_consts<T, S>(c);
    P2G<S> P;
    S aff[9];
    S nF[9];
    p2g_particle<false>(m, C, F, P, aff, st_out ? nF : (S*)nullptr);
    if (st_out) {
#pragma unroll
      for (int k = 0; k < 9; ++k) st_out[(int64_t)(15 + k) * c.ld + p] = to_prec<T>(nF[k]);
    }
    if (!ok) atomicOr(c.status, MPM_STATUS_OUT_OF_GRID);
    if (!finite(P.J)) atomicOr(c.status, MPM_STATUS_NONFINITE);
    if (ok) {
      scene = sc;
#pragma unroll
      for (int k = 0; k < 9; ++k) affine[k] = to_prec<T>(aff[k]) * c.dx;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        pm[k] = c.p_mass * v[k] - (affine[3 * k] * s.fx[0] + affine[3 * k + 1] * s.fx[1] + affine[3 * k + 2] * s.fx[2]);
    } else {
      zero_stencil(s);
    }
  }
  const long long key = ok ? cell_key(c, scene, s) : -1 - (long long)(threadIdx.x & 31);
  Node<T>* g = grid + (int64_t)scene * c.G;
  const StencilAddr A = stencil_addr(c, s);
  __shared__ typename ScatterStage<T>::type stage[kParticleThreads<S> / 32];  // one per warp
  auto* sb = &stage[threadIdx.x >> 5];
  const WarpRows rows = warp_rows(key, ok);
  flag_blocks(c, ok && rows.first, s.base, scene, flags);
  if constexpr (sizeof(T) == 4) {
    __syncwarp();  // a strided caller's previous chunk has been read
    row_addresses(*sb, rows.row, A, g);
    row_put(*sb, rows.row, pm, affine, s);
    __syncwarp();
    row_scatter<true>(*sb, rows.tails, rows.emit, c.p_mass);
  } else {
    slab_addresses(*sb, rows.row, A);
    T cx[3] = {pm[0], pm[1], pm[2]};
#pragma unroll 1
    for (int ox = 0; ox < 3; ++ox) {
      const T wx = sel3(s.w[0][0], s.w[1][0], s.w[2][0], ox);
      const int ax = sel3(A.ax[0], A.ax[1], A.ax[2], ox);
      T cy[3] = {cx[0], cx[1], cx[2]};
#pragma unroll
      for (int oy = 0; oy < 3; ++oy) {
        T cz[3] = {cy[0], cy[1], cy[2]};
        const T wxy = wx * s.w[oy][1];
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
          const T wgt = wxy * s.w[oz][2];
          sb->v[rows.row][oy * 3 + oz] = make_double2(wgt * cz[0], wgt * cz[1]);
          sb->u[rows.row][oy * 3 + oz] = make_double2(wgt * cz[2], wgt);
#pragma unroll
          for (int k = 0; k < 3; ++k) cz[k] += affine[3 * k + 2];
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) cy[k] += affine[3 * k + 1];
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) cx[k] += affine[3 * k];
      sb->base[rows.row] = g + ax;
      __syncwarp();
      slab_reduce64<true>(*sb, rows.tails, rows.emit, c.p_mass);
      __syncwarp();
    }
  }
}
// FP32: 7 CTAs of 128 threads per SM by default (at most 73 registers, no
// spill; measured 6 % faster than 6 CTAs); MB > 0 compiles the kernel for MB
// CTAs per SM instead (the autotuner's candidates, MpmTuning.p2g_ctas).
// Strided: the CTAs stride over the particle chunks (the adjoint's recompute,
// which exits at once when the grid store holds the substep; its poses were
// converted by the restore)
template <typename T, typename S, bool Strided = false, int MB = 0>
__global__ void __launch_bounds__(kParticleThreads<S>, MB > 0 ? MB : (sizeof(S) == 4 ? 7 : 16)) k_p2g(Consts<T> c, const T* __restrict__ st, T* __restrict__ st_out,
                                             const int* __restrict__ pscene, const int* __restrict__ order,
                                             Node<T>* __restrict__ grid, unsigned char* __restrict__ flags,
                                             PoseTableArgs pt,
                                             const int64_t* __restrict__ saved) {
  pdl_wait();     // forward: the frame is g2p's output; adjoint: the restore comes before
  pdl_trigger();
  if constexpr (Strided) {
    if (saved && *saved >= 0) return;  // the grids of this substep were restored from the grid store
    for (int64_t p0 = (int64_t)blockIdx.x * blockDim.x; p0 < c.n_particles; p0 += (int64_t)gridDim.x * blockDim.x)
      p2g_chunk<T, S>(c, st, st_out, pscene, order, grid, flags, p0 + threadIdx.x);
  } else {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    pose_table_fill<T>(pt, i, (int64_t)gridDim.x * blockDim.x);
    p2g_chunk<T, S>(c, st, st_out, pscene, order, grid, flags, i);
  }
}

// Tools in the compute precision, for grid_op and grid_op.grad.  The tool
// fields (primive_base.py:313-329) are converted once when the tools are set
// (k_tools_convert: tools_t[i] = Tool<T> of descriptor i).  The poses of
// frames f and f+1 are converted every substep by p2g or the adjoint's restore
// (poses_t[16 i + k]: k < 8 frame f, else frame f+1, one value per thread).
// Both kernels read them straight from global memory: the lanes of a warp
// load the same words (a broadcast), with no per-block staging, barrier or
// FP64 conversion.
template <typename T>
__global__ void __launch_bounds__(128) k_tools_convert(int n, const MpmToolDesc* __restrict__ tools,
                                                       Tool<T>* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) to_tool(tools[i], out[i]);
}
// the tools of one scene: tool[t], pose p0(t) at frame f, p1(t) at frame f+1
template <typename T>
struct SceneToolView {
  int n;
  const Tool<T>* tool;
  const Pose<T>* pose;
  MPM_DI SceneToolView(const Tool<T>* tools_t, const T* poses_t, const int* tool_off, int scene) {
    const int t0 = tool_off[scene];
    n = tool_off[scene + 1] - t0;
    tool = tools_t + t0;
    pose = reinterpret_cast<const Pose<T>*>(poses_t + 16 * (int64_t)t0);
  }
  MPM_DI const Pose<T>& p0(int t) const { return pose[2 * t]; }
  MPM_DI const Pose<T>& p1(int t) const { return pose[2 * t + 1]; }
};

// wall conditions of grid_op (mpm_simulator.py:241-260) with optional tape
template <typename T>
struct WallTape {
  T v_pre[3][3];
  bool low[3], up[3];
};
template <typename T>
MPM_DI void walls(const Consts<T>& c, const int* I, T* v, WallTape<T>* tp) {
  const int bound = 3;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (tp) {
#pragma unroll
      for (int k = 0; k < 3; ++k) tp->v_pre[d][k] = v[k];
    }
    bool low = I[d] < bound && v[d] < T(0);
    if (tp) tp->low[d] = low;
    if (low) {
      if (d != 1 || c.ground_friction == T(0)) {
        v[d] = T(0);
      } else if (c.ground_friction < T(10)) {
        T lin = v[1] + T(1e-30);
        T vit[3] = {v[0] - T(I[0]) * T(1e-30), v[1] - lin - T(I[1]) * T(1e-30), v[2] - T(I[2]) * T(1e-30)};
        T lit = len8(vit);
        T a = T(1) + quot(c.ground_friction * lin, lit);
        T fac = (T(0) < a) ? a : T(0);
#pragma unroll
        for (int k = 0; k < 3; ++k) v[k] = fac * (vit[k] + T(I[k]) * T(1e-30));
        v[1] = T(0);
      } else {
        v[0] = v[1] = v[2] = T(0);
      }
    }
    bool up = I[d] > c.n_grid - bound && v[d] > T(0);
    if (tp) tp->up[d] = up;
    if (up) v[d] = T(0);
  }
}
template <typename T>
MPM_DI void walls_vjp(const Consts<T>& c, const int* I, const WallTape<T>& tp, T* g) {
#pragma unroll
  for (int d = 2; d >= 0; --d) {
    if (tp.up[d]) g[d] = T(0);
    if (!tp.low[d]) continue;
    if (d != 1 || c.ground_friction == T(0)) {
      g[d] = T(0);
    } else if (c.ground_friction < T(10)) {
      const T* v = tp.v_pre[d];
      T lin = v[1] + T(1e-30);
      T vit[3] = {v[0] - T(I[0]) * T(1e-30), v[1] - lin - T(I[1]) * T(1e-30), v[2] - T(I[2]) * T(1e-30)};
      T lit = len8(vit);
      T a = T(1) + quot(c.ground_friction * lin, lit);
      T fac = (T(0) < a) ? a : T(0);
      const T go[3] = {g[0], T(0), g[2]};
      const T w[3] = {vit[0] + T(I[0]) * T(1e-30), vit[1] + T(I[1]) * T(1e-30), vit[2] + T(I[2]) * T(1e-30)};
      T g_fac = dot3(go, w);
      T g_vit[3] = {fac * go[0], fac * go[1], fac * go[2]};
      T g_lin = T(0), g_lit = T(0);
      if (T(0) < a) {
        g_lin = quot(g_fac * c.ground_friction, lit);
        g_lit = quot(-g_fac * c.ground_friction * lin, lit * lit);
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) g_vit[k] += quot(g_lit * vit[k], lit);
      g_lin -= g_vit[1];
      g[0] = g_vit[0];
      g[1] = g_vit[1] + g_lin;
      g[2] = g_vit[2];
    } else {
      g[0] = g[1] = g[2] = T(0);
    }
  }
}

// Grid store: the forward grids of a substep (the active blocks of the p2g
// grid and of the grid_op output) are kept so the adjoint substep restores
// them instead of recomputing p2g and grid_op (copy in k_grid_op, restore in
// k_restore).  Its free space is a bump counter, which all CTAs of grid_op read to
// see where the substep's n blocks go (-1: the store is full, the adjoint then
// recomputes); g2p, after them, moves it on and books the slot.
MPM_DI int64_t store_room(const MpmGridStore& st, int n) {
  const int64_t start = *st.bump;
  return start + n <= st.capacity ? start : -1;
}
MPM_DI void store_book(const MpmGridStore& st, int slot, int n) {
  const int64_t start = store_room(st, n);
  st.slot_start[slot] = start;
  st.slot_count[slot] = start >= 0 ? n : 0;
  if (start >= 0) *st.bump = start + n;
}

// 1 / m of a node with mass (m > 1e-12)
MPM_DI float node_rcp(float m) { return 1.f / m; }
MPM_DI double node_rcp(double m) { return rcp64_normal(m); }

// grid_op over the active blocks: one 64-thread CTA per block, grid-stride.
// store_slot >= 0: list block b of grid_in and of grid_out are also copied to
// the grid store at its next free block + b (g2p then books them; nothing when the
// store is full).  saved (may be null; the adjoint's recompute): when it
// points at a slot start >= 0 both grids were restored from the store and the
// kernel returns at once.  FP32: at least 16 CTAs per SM (64 registers, a small
// spill): with the grid-stride width of 16 CTAs per SM all of them are
// resident at once (measured 9.8 -> 9.2 us on 32 scenes against 80 registers).
// The block's nodes of grid_in are zeroed at the end; in the adjoint (zero_b given),
// where grid_op.grad still reads grid_in, those of zero_b (the velocity adjoint).
template <typename T>
__global__ void __launch_bounds__(64, sizeof(T) == 4 ? 16 : 1) k_grid_op(Consts<T> c, const int* __restrict__ active,
                                                const int* __restrict__ n_active, Node<T>* __restrict__ grid_in,
                                                Node<T>* __restrict__ grid_out, Node<T>* __restrict__ zero_b,
                                                const Tool<T>* __restrict__ tools_t, const T* __restrict__ poses_t,
                                                const int* __restrict__ tool_off, MpmGridStore store,
                                                int store_slot, const int64_t* __restrict__ saved) {
  pdl_wait();     // the grid is p2g's output
  pdl_trigger();  // g2p reads its particle rows while the grid is updated
  if (saved && *saved >= 0) return;
  const int na = *n_active;
  const int64_t start = store_slot >= 0 ? store_room(store, na) : -1;
  const Node<T> zero = {T(0), T(0), T(0), T(0)};
  for (int b = blockIdx.x; b < na; b += gridDim.x) {
    const int64_t gb = active[b];
    int I[3];
    const int scene = block_node(c, gb, threadIdx.x, I);
    const SceneToolView<T> sh(tools_t, poses_t, tool_off, scene);
    const int64_t idx = gb * 64 + threadIdx.x;
    Node<T> in = grid_in[idx];
    Node<T>* stored = start >= 0 ? reinterpret_cast<Node<T>*>(store.blocks) + ((start + b) << 7) : nullptr;
    if (stored) {
      stored[threadIdx.x] = in;
      if (threadIdx.x == 0) store.block_ids[start + b] = (int)gb;
    }
    Node<T> out = {T(0), T(0), T(0), in.w};
    if (in.w > T(1e-12)) {
      T inv = node_rcp(in.w);
      T v[3] = {inv * in.x + c.gdt[0], inv * in.y + c.gdt[1], inv * in.z + c.gdt[2]};
      const T p[3] = {T(I[0]) * c.dx, T(I[1]) * c.dx, T(I[2]) * c.dx};
      for (int t = 0; t < sh.n; ++t) tool_collide(sh.tool[t], sh.p0(t), sh.p1(t), p, c.dt, v);
      walls(c, I, v, (WallTape<T>*)nullptr);
      if (!(finite(v[0]) && finite(v[1]) && finite(v[2]))) atomicOr(c.status, MPM_STATUS_NONFINITE);
      out.x = v[0];
      out.y = v[1];
      out.z = v[2];
    }
    grid_out[idx] = out;
    if (stored) stored[64 + threadIdx.x] = out;
    (zero_b ? zero_b : grid_in)[idx] = zero;
  }
}

// sums over a stencil's line along z: l0 = sum_o w n(o), l1 = sum_o o w n(o)
template <typename T>
MPM_DI void line_sums(const Stencil<T>& s, const Node<T>& n0, const Node<T>& n1, const Node<T>& n2, T* l0, T* l1) {
  const T w0 = s.w[0][2], w1 = s.w[1][2], w2 = s.w[2][2];
  const T a0[3] = {n0.x, n0.y, n0.z}, a1[3] = {n1.x, n1.y, n1.z}, a2[3] = {n2.x, n2.y, n2.z};
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const T t1 = w1 * a1[i], t2 = w2 * a2[i];
    l0[i] = w0 * a0[i] + t1 + t2;
    l1[i] = T(2) * t2 + t1;
  }
}

// sums of g2p over the stencil's nodes, node(ox, oy, oz); writes rows 0..14 and xn
template <typename T, typename F>
MPM_DI void g2p_sums(const Consts<T>& c, T* __restrict__ st_out, int64_t p, const T* x, const Stencil<T>& s, F&& node,
                     T* xn) {
  // C = k4 sum_o wgt v(o) (o - fx)^T = k4 (m1 - nv fx^T) with m1 = sum_o wgt v(o) o^T,
  // summed axis by axis (line_sums): per component 24 operations on each of the 9
  // lines along z and 12 on each plane, where a sum over nodes took 12 per node
  T nv[3] = {T(0), T(0), T(0)}, m1[9], nC[9];
  const T k4 = T(4) * c.inv_dx;
#pragma unroll
  for (int k = 0; k < 9; ++k) m1[k] = T(0);
#pragma unroll
  for (int ox = 0; ox < 3; ++ox) {
    T p0[3] = {T(0), T(0), T(0)}, py[3] = {T(0), T(0), T(0)}, pz[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int oy = 0; oy < 3; ++oy) {
      const Node<T> n0 = node(ox, oy, 0), n1 = node(ox, oy, 1), n2 = node(ox, oy, 2);
      T l0[3], l1[3];
      line_sums(s, n0, n1, n2, l0, l1);
      const T wy = s.w[oy][1];
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        p0[i] += wy * l0[i];
        pz[i] += wy * l1[i];
        if (oy > 0) py[i] += T(oy) * wy * l0[i];
      }
    }
    const T wx = s.w[ox][0];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      nv[i] += wx * p0[i];
      if (ox > 0) m1[i * 3] += T(ox) * wx * p0[i];
      m1[i * 3 + 1] += wx * py[i];
      m1[i * 3 + 2] += wx * pz[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) nC[i * 3 + j] = k4 * (m1[i * 3 + j] - s.fx[j] * nv[i]);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    T t = x[i] + c.dt * nv[i];
    T mn = (t < c.x_hi) ? t : c.x_hi;
    xn[i] = (c.x_lo < mn) ? mn : c.x_lo;
  }
  store_row(st_out, c.ld, p, 0, 3, xn);
  store_row(st_out, c.ld, p, 3, 3, nv);
  store_row(st_out, c.ld, p, 6, 9, nC);
}

// g2p of particle p (mpm_simulator.py:265-284): writes rows 0..14 of st_out
// and xn; returns false (the state copied unchanged) for a particle whose
// stencil left the grid
template <typename T>
MPM_DI bool g2p_particle(const Consts<T>& c, const T* __restrict__ st, T* __restrict__ st_out, int64_t p, int scene,
                         const Node<T>* __restrict__ grid, T* xn) {
  T x[3];
  load_row_cg(st, c.ld, p, 0, 3, x);
  Stencil<T> s;
  if (!make_stencil(c, x, s)) {  // flagged by k_p2g; the particle keeps its state
#pragma unroll
    for (int k = 0; k < 15; ++k) st_out[(int64_t)k * c.ld + p] = __ldcg(st + (int64_t)k * c.ld + p);
    return false;
  }
  const Node<T>* g = grid + (int64_t)scene * c.G;
  const StencilAddr A = stencil_addr(c, s);
  pdl_wait();  // the grid is grid_op's output
  g2p_sums(c, st_out, p, x, s, [&](int ox, int oy, int oz) { return g[A.at(ox, oy, oz)]; }, xn);
  return true;
}
// FP32, one gather of the nodes per cell of a warp, as in g2p.grad: the lanes of a cell
// find each other by __match_any_sync, 27 lanes fetch the cell's nodes, all read them
// from shared memory.  For launches of more than one wave, where the L1's wavefronts
// bound the gathers (1.1M particles of one scene by cell 34.6 -> 30.6 us, 200,000 11.9
// -> 11.1); smaller ones wait for one warp's chain, which the grouping makes longer
// (30,000 particles in the caller's order 8.3 -> 9.6 us), so they gather lane by lane.
// So do the frames of callers that never sort them: their warps hold more cells than fit
// and gather lane by lane here too, from an L1 that the stages have halved (unsorted
// 400,000 particles 30.5 us without the stages and 38.5 with them, 1.1M 65 and 85).
struct GatherStage {
  float4 nodes[kStagedGroups][27];
  const Node<float>* base[kStagedGroups];
  int off[kStagedGroups][9];
};
MPM_DI void g2p_warp(const Consts<float>& c, const float* __restrict__ st, float* __restrict__ st_out, int64_t p, bool valid,
                     int scene, const Node<float>* __restrict__ grid, GatherStage& sb) {
  float x[3] = {0.f, 0.f, 0.f}, xn[3];
  if (valid) load_row_cg(st, c.ld, p, 0, 3, x);
  Stencil<float> s;
  zero_stencil(s);
  const bool ok = valid && make_stencil(c, x, s);
  if (valid && !ok) {
#pragma unroll
    for (int k = 0; k < 15; ++k) st_out[(int64_t)k * c.ld + p] = __ldcg(st + (int64_t)k * c.ld + p);
  }
  const Node<float>* g = grid + (int64_t)scene * c.G;
  if (!ok) zero_stencil(s);
  const StencilAddr A = stencil_addr(c, s);
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(0xffffffffu, ok ? cell_key(c, scene, s) : -1 - (long long)lane);
  const int first = __ffs(peers) - 1;
  const unsigned leaders = __ballot_sync(0xffffffffu, ok && lane == first);
  const int ng = __popc(leaders);
  pdl_wait();
  if (ng <= kStagedGroups) {
    const int mine = __popc(leaders & ((1u << first) - 1u));
    if (ok && lane == first) {
      sb.base[mine] = g;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        sb.off[mine][k] = A.ax[k];
        sb.off[mine][3 + k] = A.ay[k];
        sb.off[mine][6 + k] = A.az[k];
      }
    }
    __syncwarp();
    const int node = lane < 27 ? lane : 26, ox = node / 9, oy = node / 3 % 3, oz = node % 3;
    for (int b = 0; b < ng; b += 4) {
      float4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (b + k < ng)
          v[k] = *reinterpret_cast<const float4*>(sb.base[b + k] +
                                                  (sb.off[b + k][ox] + sb.off[b + k][3 + oy] + sb.off[b + k][6 + oz]));
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (b + k < ng && lane < 27) sb.nodes[b + k][lane] = v[k];
    }
    __syncwarp();
    if (ok)
      g2p_sums(c, st_out, p, x, s, [&](int ax, int ay, int az) {
        const float4 v = sb.nodes[mine][9 * ax + 3 * ay + az];
        return Node<float>{v.x, v.y, v.z, v.w};
      }, xn);
  } else if (ok) {
    g2p_sums(c, st_out, p, x, s, [&](int ox, int oy, int oz) { return g[A.at(ox, oy, oz)]; }, xn);
  }
}
// One thread ends the substep's block bookkeeping: it books what grid_op put into the
// grid store (store_slot >= 0) and empties the list.
// At least MB CTAs of 128 threads per SM (MpmTuning.g2p_ctas; 0 = 8 in FP32:
// at most 64 registers)
template <typename T, int MB = 0, bool Shared = false>
__global__ void __launch_bounds__(kParticleThreads<T>, MB > 0 ? MB : (sizeof(T) == 4 ? 8 : 1)) k_g2p(Consts<T> c, const T* __restrict__ st, T* __restrict__ st_out,
                                             const int* __restrict__ pscene, const Node<T>* __restrict__ grid,
                                             int* __restrict__ counter, MpmGridStore store, int store_slot) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = p < c.n_particles;
  const int scene = valid ? __ldcg(pscene + p) : 0;  // issued with x
  if constexpr (Shared) {
    __shared__ GatherStage stage[kParticleThreads<T> / 32];
    g2p_warp(c, st, st_out, p, valid, scene, grid, stage[threadIdx.x >> 5]);
  } else {
    T xn[3];
    if (valid) g2p_particle(c, st, st_out, p, scene, grid, xn);
  }
  pdl_wait();  // grid_op reads the counter (and lanes without a stencil have not waited)
  pdl_trigger();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    if (store_slot >= 0) store_book(store, store_slot, *counter);
    *counter = 0;
  }
}

// ---------------------------------------------------------------------------
// adjoint kernels
// ---------------------------------------------------------------------------
// g2p.grad: writes the x rows of g0 (partial; add: adds to them) and scatters into
// g_grid
// st1 (frame f+1, may be null): its v rows are the g2p output, so the clamp
// mask needs no second gather of the grid.
// FP32: 8 CTAs of 128 threads per SM by default (64 registers, 60 B of spill): it
// waits on its gathers (1.1M particles: 5, 6, 7, 8 CTAs 94.1, 88.3, 83.7, 83.4 us);
// MB > 0: MB CTAs per SM (MpmTuning.g2p_adj_ctas)
template <typename T, int MB = 0>
__global__ void __launch_bounds__(kParticleThreads<T>, MB > 0 ? MB : (sizeof(T) == 4 ? 8 : 8)) k_g2p_adj(Consts<T> c, const T* __restrict__ st, const T* __restrict__ st1,
                                                 const T* __restrict__ g1, T* __restrict__ g0,
                                                 const int* __restrict__ pscene, const int* __restrict__ order,
                                                 bool add, const Node<T>* __restrict__ grid,
                                                 Node<T>* __restrict__ g_grid) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < c.n_particles;  // every lane stays for the warp's scatter
  const int64_t p = particle_of(order, i, valid);
  Stencil<T> s;
  zero_stencil(s);
  bool ok = false;
  int scene = 0;
  T x[3] = {T(0), T(0), T(0)};
  T nv[3] = {T(0), T(0), T(0)};
  T gnv[3] = {T(0), T(0), T(0)}, gC[9], gx[3] = {T(0), T(0), T(0)}, gx1[3] = {T(0), T(0), T(0)};
#pragma unroll
  for (int k = 0; k < 9; ++k) gC[k] = T(0);
  if (valid) {
    // every row this particle needs is requested together with x
    load_row_cg(st, c.ld, p, 0, 3, x);
    if (st1) load_row_cg(st1, c.ld, p, 3, 3, nv);
    load_row_cg(g1, c.ld, p, 0, 3, gx1);
    load_row_cg(g1, c.ld, p, 3, 3, gnv);
    load_row_cg(g1, c.ld, p, 6, 9, gC);
    scene = __ldcg(pscene + p);
    ok = make_stencil(c, x, s);
    if (!ok) {
      zero_stencil(s);
      scene = 0;
      const T z[3] = {T(0), T(0), T(0)};
      if (!add) store_row(g0, c.ld, p, 0, 3, z);
    }
  }
  if (!ok) {  // no contribution (and no 0 * inf) from particles outside the grid
#pragma unroll
    for (int k = 0; k < 3; ++k) nv[k] = gnv[k] = gx1[k] = T(0);
#pragma unroll
    for (int k = 0; k < 9; ++k) gC[k] = T(0);
  }
  const int64_t off = (int64_t)scene * c.G;
  const Node<T>* g = grid + off;
  Node<T>* gg = g_grid + off;
  const StencilAddr A = stencil_addr(c, s);
  pdl_wait();  // the restored (or recomputed) grid and the zeroed g_grid
  pdl_trigger();
  if (ok) {
    if (!st1) {
#pragma unroll
      for (int ox = 0; ox < 3; ++ox)
#pragma unroll
        for (int oy = 0; oy < 3; ++oy)
#pragma unroll
          for (int oz = 0; oz < 3; ++oz) {
            T wgt = s.w[ox][0] * s.w[oy][1] * s.w[oz][2];
            Node<T> n = g[A.at(ox, oy, oz)];
            nv[0] += wgt * n.x;
            nv[1] += wgt * n.y;
            nv[2] += wgt * n.z;
          }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      T t = x[i] + c.dt * nv[i];
      T mn = (t < c.x_hi) ? t : c.x_hi;
      bool pass = (t < c.x_hi) && (c.x_lo < mn);
      T gt = pass ? gx1[i] : T(0);
      gx[i] = gt;
      gnv[i] += c.dt * gt;
    }
  }
  const long long key = ok ? cell_key(c, scene, s) : -1 - (long long)(threadIdx.x & 31);
  __shared__ typename ScatterStage<T>::type stage[kParticleThreads<T> / 32];  // one per warp
  auto* sb = &stage[threadIdx.x >> 5];
  const WarpRows rows = warp_rows(key, ok);
  const T k4 = T(4) * c.inv_dx;
  // the x-derivative through dp = o - fx of sum_o wgt gv(o) . (k4 gC dp) is
  // -k4 gC^T sum_o wgt gv(o) = -k4 gC^T new_v
  T gfx[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) gfx[j] = -k4 * (gC[j] * nv[0] + gC[3 + j] * nv[1] + gC[6 + j] * nv[2]);
  // u(o) = gnv + k4 gC (o - fx): the node value is wgt(o) u(o) and the weight
  // adjoint gv(o) . u(o); u is stepped across the stencil by the columns of k4 gC
  T ux[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j) gC[3 * i + j] *= k4;
    ux[i] = gnv[i] - (gC[3 * i] * s.fx[0] + gC[3 * i + 1] * s.fx[1] + gC[3 * i + 2] * s.fx[2]);
  }
  // weight adjoints h(o) = gv(o) . u(o), summed axis by axis against the weights
  // and their derivatives; the gathers of the grid velocity come before the scatter,
  // which then touches no global memory but its atomics.  FP32: the L1's wavefronts
  // bound the gathers (76 % of their peak; 27 loads of 16 B per lane from some 12
  // lines each), and the lanes of one cell read the same nodes, so 27 lanes fetch a
  // cell's nodes once into the row stage and the lanes read them there: 1.1M
  // particles 85.4 -> 83.4 us, 0.8M 64.7 -> 61.5, 30,000 19.6 -> 16.4.  A warp of more
  // cells than the stage holds gathers for itself (a loop over the cells, one copy of
  // the arithmetic, kept more registers live: 89.7 us)
  const auto gather = [&](auto&& node) {
    T dw[3][3];
    stencil_derivatives(s, dw);
    T sx = T(0), sy = T(0), sz = T(0);
    T vx[3] = {ux[0], ux[1], ux[2]};
#pragma unroll
    for (int ox = 0; ox < 3; ++ox) {
      T p0 = T(0), p1 = T(0), pz = T(0);
      T vy[3] = {vx[0], vx[1], vx[2]};
#pragma unroll
      for (int oy = 0; oy < 3; ++oy) {
        T vz[3] = {vy[0], vy[1], vy[2]};
        T l0 = T(0), lz = T(0);
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
          const Node<T> n = node(ox, oy, oz);
          const T gv[3] = {n.x, n.y, n.z};
          const T h = dot3(gv, vz);
          l0 += s.w[oz][2] * h;
          lz += dw[oz][2] * h;
#pragma unroll
          for (int i = 0; i < 3; ++i) vz[i] += gC[3 * i + 2];
        }
        p0 += s.w[oy][1] * l0;
        p1 += dw[oy][1] * l0;
        pz += s.w[oy][1] * lz;
#pragma unroll
        for (int i = 0; i < 3; ++i) vy[i] += gC[3 * i + 1];
      }
      sx += dw[ox][0] * p0;
      sy += s.w[ox][0] * p1;
      sz += s.w[ox][0] * pz;
#pragma unroll
      for (int i = 0; i < 3; ++i) vx[i] += gC[3 * i];
    }
    gfx[0] += sx;
    gfx[1] += sy;
    gfx[2] += sz;
  };
  if constexpr (sizeof(T) == 4) {
    row_addresses(*sb, rows.row, A, gg);
    __syncwarp();
    if (__popc(rows.emit) <= kStagedGroups) {  // the same for the whole warp
      const int lane = threadIdx.x & 31, node = lane < 27 ? lane : 26;
      const int ox = node / 9, oy = node / 3 % 3, oz = node % 3;
      unsigned m = rows.emit;
      for (int b = 0; b < kStagedGroups && m; b += 4) {
        float4 v[4];
        unsigned left = m;
#pragma unroll
        for (int k = 0; k < 4; ++k) {  // four loads in flight
          if (left) {
            const int r = __ffs(left) - 1;
            left &= left - 1u;
            v[k] = *reinterpret_cast<const float4*>(grid + (sb->base[r] - g_grid) +
                                                    (sb->off[r][ox] + sb->off[r][3 + oy] + sb->off[r][6 + oz]));
          }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (m) {
            m &= m - 1u;
            if (lane < 27) sb->nodes[b + k][lane] = v[k];
          }
        }
      }
      __syncwarp();
      const float4* mine = sb->nodes[ok ? __popc(rows.emit & ((1u << rows.row) - 1u)) : 0];
      if (ok)
        gather([&](int ax, int ay, int az) {
          const float4 v = mine[9 * ax + 3 * ay + az];
          return Node<T>{v.x, v.y, v.z, v.w};
        });
      __syncwarp();
    } else if (ok) {
      gather([&](int ax, int ay, int az) { return g[A.at(ax, ay, az)]; });
    }
  } else if (ok) {
    gather([&](int ax, int ay, int az) { return g[A.at(ax, ay, az)]; });
  }
  if constexpr (sizeof(T) == 4) {
    row_put(*sb, rows.row, ux, gC, s);
    __syncwarp();
    row_scatter<false>(*sb, rows.tails, rows.emit, 0.f);
  } else {
    slab_addresses(*sb, rows.row, A);
#pragma unroll 1
    for (int ox = 0; ox < 3; ++ox) {
      const T wx = sel3(s.w[0][0], s.w[1][0], s.w[2][0], ox);
      const int ax = sel3(A.ax[0], A.ax[1], A.ax[2], ox);
      T uy[3] = {ux[0], ux[1], ux[2]};
#pragma unroll
      for (int oy = 0; oy < 3; ++oy) {
        T uz[3] = {uy[0], uy[1], uy[2]};
        const T wxy = wx * s.w[oy][1];
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
          const T wgt = wxy * s.w[oz][2];
          sb->v[rows.row][oy * 3 + oz] = make_double2(wgt * uz[0], wgt * uz[1]);
          sb->u[rows.row][oy * 3 + oz] = make_double2(wgt * uz[2], 0.0);
#pragma unroll
          for (int i = 0; i < 3; ++i) uz[i] += gC[3 * i + 2];
        }
#pragma unroll
        for (int i = 0; i < 3; ++i) uy[i] += gC[3 * i + 1];
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) ux[i] += gC[3 * i];
      sb->base[rows.row] = gg + ax;
      __syncwarp();
      slab_reduce64<false>(*sb, rows.tails, rows.emit, 1.0);
      __syncwarp();
    }
  }
  if (ok) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      gx[d] += c.inv_dx * gfx[d];
      if (add) gx[d] += g0[(int64_t)d * c.ld + p];
    }
    store_row(g0, c.ld, p, 0, 3, gx);
  }
}

// grid_op.grad over the active blocks: g_grid (velocity adjoint) -> g_in
// (mv.xyz, m); tool-pose gradients of frames f and f+1 reduced per warp in
// FP64 and added with one atomic per warp and component.
// Sums 16 values over the 32 lanes of a warp by recursive halving
// (reduce-scatter): each level sends half of the values still held to the
// partner lane and keeps the other half, 16 shuffles in all instead of 80
// for 16 butterfly all-reduces.  Returns the full sum of value k (set on
// return, from lane bits 4..1); lanes 2j and 2j+1 hold the same k.
template <typename T>
MPM_DI T warp_reduce_scatter16(T (&v)[16], int& k) {
  const int lane = threadIdx.x & 31;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4, h1 = lane & 2;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const T send = h4 ? v[i] : v[i + 8];
    const T keep = h4 ? v[i + 8] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const T send = h3 ? v[i] : v[i + 4];
    const T keep = h3 ? v[i + 4] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const T send = h2 ? v[i] : v[i + 2];
    const T keep = h2 ? v[i + 2] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  {
    const T send = h1 ? v[0] : v[1];
    const T keep = h1 ? v[1] : v[0];
    v[0] = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  }
  k = (h4 ? 8 : 0) + (h3 ? 4 : 0) + (h2 ? 2 : 0) + (h1 ? 1 : 0);
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// When saved points at a slot start >= 0 (the grid store holds the substep), the p2g
// grid's nodes are read from the store and grid_in, which was not restored, stays
// zero; else grid_in's listed blocks are zeroed here, by their last reader.
// At least MB CTAs of 64 threads per SM (MpmTuning.grid_op_adj_ctas; 0 = 6:
// at most 168 registers)
template <typename T, int MB = 0>
__global__ void __launch_bounds__(64, MB > 0 ? MB : (sizeof(T) == 4 ? 6 : 1)) k_grid_op_adj(Consts<T> c, const int* __restrict__ active,
                                                    const int* __restrict__ n_active,
                                                    Node<T>* __restrict__ grid_in,
                                                    const Node<T>* __restrict__ g_grid, Node<T>* __restrict__ g_in,
                                                    const Tool<T>* __restrict__ tools_t,
                                                    const T* __restrict__ poses_t, const int* __restrict__ tool_off,
                                                    const void* __restrict__ kept, const int64_t* __restrict__ saved,
                                                    double* __restrict__ g_pose_f, double* __restrict__ g_pose_f1) {
  pdl_wait();     // g_grid is g2p.grad's output
  pdl_trigger();  // p2g.grad recomputes its particles' stress meanwhile
  const int na = *n_active;
  const int64_t start = saved ? *saved : -1;
  for (int b = blockIdx.x; b < na; b += gridDim.x) {
    const int64_t gb = active[b];
    int I[3];
    const int scene = block_node(c, gb, threadIdx.x, I);
    const SceneToolView<T> sh(tools_t, poses_t, tool_off, scene);
    const int64_t idx = gb * 64 + threadIdx.x;
    const Node<T>* from =
        start >= 0 ? reinterpret_cast<const Node<T>*>(kept) + ((start + b) << 7) + threadIdx.x : grid_in + idx;
    const Node<T> in = *from;
    Node<T> go = g_grid[idx];
    const bool active_node = in.w > T(1e-12) && (go.x != T(0) || go.y != T(0) || go.z != T(0));
    const T p[3] = {T(I[0]) * c.dx, T(I[1]) * c.dx, T(I[2]) * c.dx};
    T vt[MAX_TOOLS_PER_SCENE + 1][3];
    WallTape<T> wt;
    T g[3] = {go.x, go.y, go.z};
    const T inv = active_node ? node_rcp(in.w) : T(0);
    unsigned hits = 0u;  // bit t: tool t is in contact with this node
    if (active_node) {
      T v[3] = {inv * in.x + c.gdt[0], inv * in.y + c.gdt[1], inv * in.z + c.gdt[2]};
      for (int t = 0; t < sh.n; ++t) {
#pragma unroll
        for (int k = 0; k < 3; ++k) vt[t][k] = v[k];
        if (tool_collide(sh.tool[t], sh.p0(t), sh.p1(t), p, c.dt, v)) hits |= 1u << t;
      }
      walls(c, I, v, &wt);
      walls_vjp(c, I, wt, g);
    }
    const int t0 = tool_off[scene];
    for (int t = sh.n - 1; t >= 0; --t) {
      const bool hit = (hits >> t) & 1u;  // without contact g passes unchanged
      if (!__any_sync(0xffffffffu, hit)) continue;
      PoseGrad<T> g0, g1;
      g0.zero();
      g1.zero();
      if (hit) tool_collide_vjp(sh.tool[t], sh.p0(t), sh.p1(t), p, c.dt, vt[t], g, g0, g1);
      double* d0 = g_pose_f + 8 * (t0 + t);
      double* d1 = g_pose_f1 + 8 * (t0 + t);
      T v16[16] = {g0.pos[0], g0.pos[1], g0.pos[2], g0.rot[0], g0.rot[1], g0.rot[2], g0.rot[3], g0.gap,
                   g1.pos[0], g1.pos[1], g1.pos[2], g1.rot[0], g1.rot[1], g1.rot[2], g1.rot[3], g1.gap};
      int k;
      const T v = warp_reduce_scatter16(v16, k);
      if ((threadIdx.x & 1) == 0 && v != T(0)) atomicAdd((k < 8 ? d0 + k : d1 + (k - 8)), double(v));
    }
    Node<T> res = {T(0), T(0), T(0), T(0)};
    if (active_node) {
      res.x = g[0] * inv;
      res.y = g[1] * inv;
      res.z = g[2] * inv;
      res.w = -(g[0] * in.x + g[1] * in.y + g[2] * in.z) * inv * inv;
    }
    g_in[idx] = res;
    if (start < 0) grid_in[idx] = Node<T>{T(0), T(0), T(0), T(0)};
  }
}

// p2g.grad + svd_grad + compute_F_tmp.grad: gathers g_in; reads the partial
// x gradient left in g0 by k_g2p_adj and writes all 24 rows of g0 (add: adds to
// rows 3..23; k_g2p_adj already added rows 0..2 to theirs).
// FP32: 4 CTAs of 128 threads per SM by default (128 registers, 88 B of spill stores and
// 108 of loads; 1.1M particles: 4, 5, 6 CTAs 112.7, 118.8, 130.0 us, the latter spilling
// 444 / 572 and 632 / 744 B); MB > 0: MB CTAs per SM (MpmTuning.p2g_adj_ctas)
template <typename T, typename S, int MB = 0>
__global__ void __launch_bounds__(kParticleThreads<S>, MB > 0 ? MB : (sizeof(S) == 4 ? 4 : 8)) k_p2g_adj(Consts<T> c, const T* __restrict__ st, const T* __restrict__ g1,
                                                 T* __restrict__ g0, const int* __restrict__ pscene, bool add,
                                                 const Node<T>* __restrict__ g_in) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= c.n_particles) return;
  // the adjoint rows read after the forward recompute and the gather are
  // fetched into L2 now, so those later loads do not wait on DRAM
#pragma unroll
  for (int k = 0; k < 3; ++k) prefetch_l2(g0 + (int64_t)k * c.ld + p);
#pragma unroll
  for (int k = 15; k < 24; ++k) prefetch_l2(g1 + (int64_t)k * c.ld + p);
  T x[3], v[3];
  S C[9], F[9];
  load_row_cg(st, c.ld, p, 0, 3, x);
  load_row_cg(st, c.ld, p, 3, 3, v);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    C[k] = to_prec<S>(__ldcg(st + (int64_t)(6 + k) * c.ld + p));
    F[k] = to_prec<S>(__ldcg(st + (int64_t)(15 + k) * c.ld + p));
  }
  const int scene = __ldcg(pscene + p);  // issued with the state rows
  Stencil<T> s;
  bool ok = make_stencil(c, x, s);
  const MatConsts<S>& m = mat_consts<T, S>(c);
  P2G<S> P;
  S aff[9];
  p2g_particle<true>(m, C, F, P, aff, (S*)nullptr);
  T affine[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) affine[k] = to_prec<T>(aff[k]);
  T gx[3], gv[3] = {T(0), T(0), T(0)};
  load_row_cg(g0, c.ld, p, 0, 3, gx);
  S g_aff[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) g_aff[k] = S(0);
  pdl_wait();  // g_in is grid_op.grad's output
  pdl_trigger();
  if (ok) {
    const Node<T>* gg = g_in + (int64_t)scene * c.G;
    const StencilAddr A = stencil_addr(c, s);
    T ga[9], dw[3][3];
    stencil_derivatives(s, dw);
#pragma unroll
    for (int k = 0; k < 9; ++k) ga[k] = T(0);
    // q(o) = wgt(o) gn(o) and sq = sum_o q(o): the adjoints of m v (gv = m sq) and of
    // dp = (o - fx) dx through A dp (gfx = -dx A^T sq) need only the sum; the adjoint
    // of A (ga = sum_o q dp^T) takes sum_o q o^T, and the weights' adjoints
    // h(o) = gn(o) . (m v + A dp) + gm(o) m their sums against the weights and their
    // derivatives.  All are summed axis by axis; the node value m v + A dp is
    // stepped across the stencil by the columns of dx A
    T sq[3] = {T(0), T(0), T(0)}, sx = T(0), sy = T(0), sz = T(0);
    T ad[9], cx[3];
#pragma unroll
    for (int k = 0; k < 9; ++k) ad[k] = affine[k] * c.dx;
#pragma unroll
    for (int k = 0; k < 3; ++k) cx[k] = c.p_mass * v[k] - (ad[3 * k] * s.fx[0] + ad[3 * k + 1] * s.fx[1] + ad[3 * k + 2] * s.fx[2]);
#pragma unroll
    for (int ox = 0; ox < 3; ++ox) {
      T p0[3] = {T(0), T(0), T(0)}, py[3] = {T(0), T(0), T(0)}, pz[3] = {T(0), T(0), T(0)};
      T h0 = T(0), h1 = T(0), hz = T(0);
      T cy[3] = {cx[0], cx[1], cx[2]};
#pragma unroll
      for (int oy = 0; oy < 3; ++oy) {
        T cz[3] = {cy[0], cy[1], cy[2]};
        const Node<T> n[3] = {gg[A.at(ox, oy, 0)], gg[A.at(ox, oy, 1)], gg[A.at(ox, oy, 2)]};
        T l0[3], l1[3], m0 = T(0), mz = T(0);
        line_sums(s, n[0], n[1], n[2], l0, l1);
#pragma unroll
        for (int oz = 0; oz < 3; ++oz) {
          const T gn[3] = {n[oz].x, n[oz].y, n[oz].z};
          const T h = dot3(gn, cz) + n[oz].w * c.p_mass;
          m0 += s.w[oz][2] * h;
          mz += dw[oz][2] * h;
#pragma unroll
          for (int k = 0; k < 3; ++k) cz[k] += ad[3 * k + 2];
        }
        const T wy = s.w[oy][1];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          p0[k] += wy * l0[k];
          pz[k] += wy * l1[k];
          if (oy > 0) py[k] += T(oy) * wy * l0[k];
        }
        h0 += wy * m0;
        h1 += dw[oy][1] * m0;
        hz += wy * mz;
#pragma unroll
        for (int k = 0; k < 3; ++k) cy[k] += ad[3 * k + 1];
      }
      const T wx = s.w[ox][0];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        sq[k] += wx * p0[k];
        if (ox > 0) ga[3 * k] += T(ox) * wx * p0[k];
        ga[3 * k + 1] += wx * py[k];
        ga[3 * k + 2] += wx * pz[k];
      }
      sx += dw[ox][0] * h0;
      sy += wx * h1;
      sz += wx * hz;
#pragma unroll
      for (int k = 0; k < 3; ++k) cx[k] += ad[3 * k];
    }
    // ga = sum_o q (o - fx)^T dx from its accumulated sum_o q o^T
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
      for (int j = 0; j < 3; ++j) ga[3 * k + j] = c.dx * (ga[3 * k + j] - s.fx[j] * sq[k]);
    T gfx[3] = {sx, sy, sz};
#pragma unroll
    for (int j = 0; j < 3; ++j) gfx[j] -= ad[j] * sq[0] + ad[3 + j] * sq[1] + ad[6 + j] * sq[2];
#pragma unroll
    for (int k = 0; k < 3; ++k) gv[k] = c.p_mass * sq[k];
#pragma unroll
    for (int d = 0; d < 3; ++d) gx[d] += c.inv_dx * gfx[d];
#pragma unroll
    for (int k = 0; k < 9; ++k) g_aff[k] = to_prec<S>(ga[k]);
  }
  S gF1[9], gC[9], gF[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) gF1[k] = to_prec<S>(g1[(int64_t)(15 + k) * c.ld + p]);
  p2g_particle_vjp(m, C, F, P, g_aff, gF1, gC, gF);
  T out[21];
#pragma unroll
  for (int k = 0; k < 3; ++k) out[k] = gv[k];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    out[3 + k] = to_prec<T>(gC[k]);
    out[12 + k] = to_prec<T>(gF[k]);
  }
  if (add) {  // all 21 loads before the first store
    T old[21];
    load_row_cg(g0, c.ld, p, 3, 21, old);
#pragma unroll
    for (int k = 0; k < 21; ++k) out[k] += old[k];
  }
  store_row(g0, c.ld, p, 0, 3, gx);
  store_row(g0, c.ld, p, 3, 21, out);
}

// ---------------------------------------------------------------------------
// start of an adjoint substep
// ---------------------------------------------------------------------------
// Converts the substep's tool poses, and when the grid store's slot holds the
// substep, restores the active list, its length and grid a_out (grid_op output) and
// zeroes the same blocks of grid b (the velocity adjoint); grid_op.grad, the one
// reader of the p2g grid, takes that from the store (an iteration of 64 scenes,
// 1.1M particles: 35.9 -> 34.7 ms, restoring it too cost 10 us a substep).
// Otherwise it empties the list, for the p2g that follows.  Grid-stride.
template <typename T>
__global__ void __launch_bounds__(256) k_restore(int* __restrict__ counter, MpmGridStore store, int slot,
                                                 int* __restrict__ active, Node<T>* __restrict__ a_out, Node<T>* __restrict__ b,
                                                 PoseTableArgs pt) {
  pdl_wait();
  pdl_trigger();
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  pose_table_fill<T>(pt, i0, stride);
  const int64_t start = slot >= 0 ? store.slot_start[slot] : -1;
  const int cnt = start >= 0 ? store.slot_count[slot] : 0;
  if (i0 == 0) *counter = cnt;
  const Node<T>* src = reinterpret_cast<const Node<T>*>(store.blocks);
  const Node<T> z = {T(0), T(0), T(0), T(0)};
  for (int64_t i = i0; i < (int64_t)cnt * 64; i += stride) {
    const int blk = store.block_ids[start + (i >> 6)];
    if ((i & 63) == 0) active[i >> 6] = blk;
    const Node<T>* sb = src + ((start + (i >> 6)) << 7) + (i & 63);
    a_out[(int64_t)blk * 64 + (i & 63)] = sb[64];
    b[(int64_t)blk * 64 + (i & 63)] = z;
  }
}

// The list of flagged blocks, in runs of consecutive blocks (the order of the runs is
// not significant), and the flags cleared: 16 flags per thread.  saved (may be
// null): nothing to do when the grid store held the substep.
template <typename T>
__global__ void __launch_bounds__(128) k_list_blocks(unsigned char* __restrict__ flags, int64_t total,
                                                     int* __restrict__ active, int* __restrict__ counter,
                                                     const int64_t* __restrict__ saved) {
  pdl_wait();
  pdl_trigger();
  if (saved && *saved >= 0) return;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t first = 16 * i;
  uint4 f = make_uint4(0u, 0u, 0u, 0u);
  if (first < total) {  // the flag buffer is padded to 16 bytes with zeros
    uint4* at = reinterpret_cast<uint4*>(flags) + i;
    f = *at;
    if (f.x | f.y | f.z | f.w) *at = make_uint4(0u, 0u, 0u, 0u);
  }
  const unsigned w[4] = {f.x, f.y, f.z, f.w};  // bytes 0 or 1
  int mine = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) mine += __popc(w[k]);
  const int lane = threadIdx.x & 31;
  int upto = mine;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, upto, d);
    if (lane >= d) upto += t;
  }
  const int all = __shfl_sync(0xffffffffu, upto, 31);
  if (all == 0) return;
  int at = 0;
  if (lane == 0) at = atomicAdd(counter, all);
  at = __shfl_sync(0xffffffffu, at, 0) + upto - mine;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    for (unsigned m = w[k]; m; m &= m - 1u) active[at++] = (int)(first + 4 * k + ((__ffs(m) - 1) >> 3));
}

// ---------------------------------------------------------------------------
// per-particle tool terms (contact losses, tool distances)
// ---------------------------------------------------------------------------
// The tools of the scene of a CTA's first particle in the compute precision,
// converted once per CTA: a thread that converts a descriptor and a pose itself
// takes some 35 FP64 conversions per tool, on the pipe that issues one
// instruction every 16 cycles.  A particle of another scene (a CTA that
// straddles scenes) still converts its own.
template <typename T>
struct StagedTools {
  int scene, t0, n;
  Tool<T> tool[MAX_TOOLS_PER_SCENE];
  Pose<T> pose[MAX_TOOLS_PER_SCENE];
};
// all threads of the CTA; `first`: the CTA's first particle (in range)
template <typename T>
MPM_DI void stage_tools(StagedTools<T>& sh, const int* __restrict__ pscene, int64_t first,
                        const MpmToolDesc* __restrict__ tools, const int* __restrict__ tool_off,
                        const double* __restrict__ pose) {
  const int sc = pscene[first];
  const int t0 = tool_off[sc], n = tool_off[sc + 1] - t0;
  if (threadIdx.x == 0) {
    sh.scene = sc;
    sh.t0 = t0;
    sh.n = n;
  }
  if ((int)threadIdx.x < n) {
    to_tool(tools[t0 + threadIdx.x], sh.tool[threadIdx.x]);
    to_pose(pose + 8 * (t0 + threadIdx.x), sh.pose[threadIdx.x]);
  }
  __syncthreads();
}
template <typename T>
MPM_DI void staged_tool(const StagedTools<T>& sh, int scene, int t, const MpmToolDesc* __restrict__ tools,
                        const double* __restrict__ pose, Tool<T>& tl, Pose<T>& P) {
  if (scene == sh.scene) {
    tl = sh.tool[t - sh.t0];
    P = sh.pose[t - sh.t0];
  } else {
    to_tool(tools[t], tl);
    to_pose(pose + 8 * t, P);
  }
}
// whether the valid lanes of a warp are of one scene (then the scene of lane 0,
// which is valid whenever any lane is): their sums go to memory once per warp
MPM_DI bool one_scene(bool valid, int scene) {
  const int s0 = __shfl_sync(0xffffffffu, scene, 0);
  return __all_sync(0xffffffffu, !valid || scene == s0);
}
// Adds 8 values of every lane to dst[0..7] in FP64: per warp (all 32 lanes, one
// atomic per value; reduce-scatter, 9 additions per lane) or per lane.  One
// atomic per particle and value made these kernels wait on the 8 addresses of a
// tool (30,000 particles: tool distance adjoint 261 us per call).
MPM_DI void add8(double* dst, double (&v)[8], bool per_warp) {
  if (!per_warp) {
    for (int k = 0; k < 8; ++k)
      if (v[k] != 0.0) atomicAdd(dst + k, v[k]);
    return;
  }
  const int lane = threadIdx.x & 31;
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const double send = h4 ? v[i] : v[i + 4];
    v[i] = (h4 ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double send = h3 ? v[i] : v[i + 2];
    v[i] = (h3 ? v[i + 2] : v[i]) + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  const double send = h2 ? v[0] : v[1];
  double s = (h2 ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, send, 4);
  s += __shfl_xor_sync(0xffffffffu, s, 2);
  s += __shfl_xor_sync(0xffffffffu, s, 1);
  const int k = (h4 ? 4 : 0) + (h3 ? 2 : 0) + (h2 ? 1 : 0);
  if ((lane & 3) == 0 && s != 0.0) atomicAdd(dst + k, s);
}
template <typename T>
MPM_DI void pose_values(const PoseGrad<T>& g, double (&v)[8]) {
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = to_prec<double>(g.pos[k]);
#pragma unroll
  for (int k = 0; k < 4; ++k) v[3 + k] = to_prec<double>(g.rot[k]);
  v[7] = to_prec<double>(g.gap);
}

// ---------------------------------------------------------------------------
// density grid and losses
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_grid_mass(Consts<T> c, const T* __restrict__ st,
                                                   const int* __restrict__ pscene, T* __restrict__ gm) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= c.n_particles) return;
  T x[3];
  load_row(st, c.ld, p, 0, 3, x);
  Stencil<T> s;
  if (!make_stencil(c, x, s)) {
    atomicOr(c.status, MPM_STATUS_OUT_OF_GRID);
    return;
  }
  T* g = gm + (int64_t)pscene[p] * c.G;
#pragma unroll
  for (int ox = 0; ox < 3; ++ox)
#pragma unroll
    for (int oy = 0; oy < 3; ++oy)
#pragma unroll
      for (int oz = 0; oz < 3; ++oz)
        atomicAdd(g + node_of(c, s, ox, oy, oz), s.w[ox][0] * s.w[oy][1] * s.w[oz][2] * c.p_mass);
}
template <typename T>
__global__ void __launch_bounds__(128) k_grid_mass_adj(Consts<T> c, const T* __restrict__ st,
                                                       const int* __restrict__ pscene, const T* __restrict__ ggm,
                                                       T* __restrict__ gst) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= c.n_particles) return;
  T x[3];
  load_row(st, c.ld, p, 0, 3, x);
  Stencil<T> s;
  if (!make_stencil(c, x, s)) return;
  const T* g = ggm + (int64_t)pscene[p] * c.G;
  T gw[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) gw[a][b] = T(0);
#pragma unroll
  for (int ox = 0; ox < 3; ++ox)
#pragma unroll
    for (int oy = 0; oy < 3; ++oy)
#pragma unroll
      for (int oz = 0; oz < 3; ++oz) {
        T gg = g[node_of(c, s, ox, oy, oz)] * c.p_mass;
        gw[ox][0] += gg * s.w[oy][1] * s.w[oz][2];
        gw[oy][1] += gg * s.w[ox][0] * s.w[oz][2];
        gw[oz][2] += gg * s.w[ox][0] * s.w[oy][1];
      }
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    T gfx = T(0);
#pragma unroll
    for (int k = 0; k < 3; ++k) gfx += gw[k][d] * dweight(s, k, d);
    gst[(int64_t)d * c.ld + p] += c.inv_dx * gfx;
  }
}
// per-scene sum |m - target| in FP64; blocks never straddle scenes
template <typename T>
__global__ void __launch_bounds__(256) k_density_l1(int64_t G, const T* __restrict__ gm, const T* __restrict__ tgt,
                                                    double weight, double* __restrict__ loss, T* __restrict__ ggm,
                                                    int blocks_per_scene) {
  int scene = blockIdx.x / blocks_per_scene;
  int b = blockIdx.x % blocks_per_scene;
  const T* a = gm + (int64_t)scene * G;
  const T* t = tgt + (int64_t)scene * G;
  double acc = 0.0;
  for (int64_t i = (int64_t)b * blockDim.x + threadIdx.x; i < G; i += (int64_t)blocks_per_scene * blockDim.x) {
    T d = a[i] - t[i];
    acc += fabs(double(d));
    if (ggm) ggm[(int64_t)scene * G + i] = T(weight) * sgn(d);
  }
  __shared__ double red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    atomicAdd(loss + scene, weight * s);
  }
}

}  // namespace mpm
