// Forward launchers: substep (p2g -> grid_op -> g2p), density grid, density
// L1 loss and the soft tool-contact distance, for the three precision modes.
#include <type_traits>

#include "mpm_kernels.cuh"
#include "mpm_launch.h"

namespace mpm {

template <typename T>
Consts<T> make_consts(const LaunchCtx& L) {
  const MpmParams& p = *L.p;
  Consts<T> c;
  c.n_grid = p.n_grid;
  c.n_scenes = p.n_scenes;
  c.n_particles = p.n_particles;
  c.ld = p.ld;
  c.G = L.G;
  c.nb = p.n_grid / 4;
  c.NB3 = (int64_t)c.nb * c.nb * c.nb;
  c.dx = T(p.dx);
  c.inv_dx = T(p.inv_dx);
  c.dt = T(p.dt);
  c.p_mass = T(p.p_mass);
  c.p_vol = T(p.p_vol);
  c.mu = T(p.mu);
  c.lam = T(p.lam);
  c.yield_stress = T(p.yield_stress);
  c.ks = T(-p.dt * p.p_vol * 4 * p.inv_dx * p.inv_dx);
  for (int k = 0; k < 3; ++k) c.gdt[k] = T(p.dt * p.gravity[k] * 30);
  c.ground_friction = T(p.ground_friction);
  c.x_lo = T(p.lower_bound * p.dx);
  c.x_hi = T(1.0 - 3 * p.dx);
  c.status = L.status;
  auto fill = [&](auto& m) {
    using S = std::decay_t<decltype(m.dt)>;
    const double mu2 = 2.0 * double(c.mu);
    m.dt = S(c.dt);
    m.p_mass = S(c.p_mass);
    m.mu2ks = S(mu2 * double(c.ks));
    m.lamks = S(double(c.lam) * double(c.ks));
    m.ysm = S(double(c.yield_stress) / mu2);
  };
  fill(c.m32);
  fill(c.m64);
  return c;
}
template Consts<float> make_consts<float>(const LaunchCtx&);
template Consts<double> make_consts<double>(const LaunchCtx&);

// The list length has a word of its own for the forward substep (g2p empties it) and
// for the adjoint (k_restore does): with a pipelined adjoint the next
// substep's list begins before this one's last kernel ends.
int* list_counter(const LaunchCtx& L, bool adjoint) { return reinterpret_cast<int*>(L.blockbuf) + (adjoint ? 1 : 0); }
// flags to list; 2,048 blocks per CTA
template <typename T>
cudaError_t launch_list_blocks(const LaunchCtx& L, const Consts<T>& c, int* counter, const int64_t* saved) {
  const int64_t total = (int64_t)c.n_scenes * c.NB3;
  MPM_LAUNCH_PDL(L, MPM_K_CLEAR, k_list_blocks<T>, (unsigned)((total + 2047) / 2048), 128, L.blockbuf + 16, total,
                 L.active, counter, saved);
  return cudaSuccess;
}
template cudaError_t launch_list_blocks<float>(const LaunchCtx&, const Consts<float>&, int*, const int64_t*);
template cudaError_t launch_list_blocks<double>(const LaunchCtx&, const Consts<double>&, int*, const int64_t*);

static inline unsigned blocks_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

size_t tools_t_bytes(int64_t n_tools) { return (size_t)(n_tools > 0 ? n_tools : 1) * sizeof(Tool<double>); }
size_t poses_t_bytes(int64_t n_tools) { return (size_t)(n_tools > 0 ? n_tools : 1) * 16 * sizeof(double); }
cudaError_t convert_tools(int precision, int n, const MpmToolDesc* tools, void* tools_t, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const unsigned g = blocks_for(n, 128);
  if (precision == MPM_PREC_FP64)
    k_tools_convert<double><<<g, 128, 0, s>>>(n, tools, (Tool<double>*)tools_t);
  else
    k_tools_convert<float><<<g, 128, 0, s>>>(n, tools, (Tool<float>*)tools_t);
  return cudaGetLastError();
}

unsigned grid_blocks_launch(const LaunchCtx& L, int64_t total_blocks) {
  const int per_sm = L.tune.grid_ctas_per_sm > 0 ? L.tune.grid_ctas_per_sm : 16;
  int64_t g = (int64_t)L.sm_count * per_sm;
  return (unsigned)(g < total_blocks ? g : (total_blocks > 0 ? total_blocks : 1));
}

template <typename T, typename S>
cudaError_t launch_substep_fwd(const LaunchCtx& L, const T* st0, T* st1, const double* pose_f,
                               const double* pose_f1, const MpmGridStore* store, int slot) {
  Consts<T> c = make_consts<T>(L);
  if (c.n_particles == 0) return cudaSuccess;  // no mass on the grid, nothing to move
  Node<T>* gin = (Node<T>*)L.grid_a;
  Node<T>* gout = (Node<T>*)L.grid_b;
  int* counter = list_counter(L, false);
  unsigned char* flags = L.blockbuf + 16;
  const int64_t* none = nullptr;
  const MpmGridStore keep = store ? *store : MpmGridStore{};
  const int keep_slot = store ? slot : -1;
  {
    constexpr int bs = kParticleThreads<S>;
    const unsigned pb = blocks_for(c.n_particles, bs);
    const PoseTableArgs pt{L.n_tools, pose_f, pose_f1, L.poses_t};
    // FP32: the CTAs-per-SM variant the tuning selects
    const int v = sizeof(S) == 4 ? L.tune.p2g_ctas : 0;
#define MPM_P2G(KERNEL) \
  MPM_LAUNCH_PDL(L, MPM_K_P2G, KERNEL, pb, bs, c, st0, st1, L.pscene, L.order, gin, flags, pt, none)
    if constexpr (sizeof(S) == 4) {
      if (v == 6)
        MPM_P2G((k_p2g<T, S, false, 6>));
      else if (v == 8)
        MPM_P2G((k_p2g<T, S, false, 8>));
      else
        MPM_P2G((k_p2g<T, S>));
    } else {
      (void)v;
      MPM_P2G((k_p2g<T, S>));
    }
#undef MPM_P2G
  }
  const cudaError_t e = launch_list_blocks<T>(L, c, counter, none);
  if (e != cudaSuccess) return e;
  MPM_LAUNCH_PDL(L, MPM_K_GRID_OP, k_grid_op<T>, grid_blocks_launch(L, (int64_t)c.n_scenes * c.NB3), 64, c,
                 (const int*)L.active, (const int*)counter, gin, gout, (Node<T>*)nullptr, (const Tool<T>*)L.tools_t,
                 (const T*)L.poses_t, L.tool_off, keep, keep_slot, none);
  {
    constexpr int bs = kParticleThreads<T>;
    const unsigned pb = blocks_for(c.n_particles, bs);
    const int v = sizeof(T) == 4 ? L.tune.g2p_ctas : 0;
#define MPM_G2P(KERNEL) \
  MPM_LAUNCH_PDL(L, MPM_K_G2P, KERNEL, pb, bs, c, st0, st1, L.pscene, gout, counter, keep, keep_slot)
    if constexpr (sizeof(T) == 4) {
      if (v == 10)
        MPM_G2P((k_g2p<T, 10>));
      else if (v == 12)
        MPM_G2P((k_g2p<T, 12>));
      else if (L.sorted && !L.order && c.n_particles > (int64_t)8 * bs * L.sm_count)
        // more than a wave of CTAs, of a caller that re-sorts its frames (measured at the kernel)
        MPM_G2P((k_g2p<T, 0, true>));
      else
        MPM_G2P(k_g2p<T>);
    } else {
      (void)v;
      MPM_G2P(k_g2p<T>);
    }
#undef MPM_G2P
  }
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_grid_mass(const LaunchCtx& L, const T* st, T* gm) {
  Consts<T> c = make_consts<T>(L);
  MPM_MEMSET(L, gm, (int64_t)c.n_scenes * c.G * sizeof(T));
  if (c.n_particles > 0)
    MPM_LAUNCH(L, MPM_K_OTHER, k_grid_mass<T>, blocks_for(c.n_particles, 128), 128, c, st, L.pscene, gm);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_grid_mass_bwd(const LaunchCtx& L, const T* st, const T* ggm, T* gst) {
  Consts<T> c = make_consts<T>(L);
  if (c.n_particles > 0)
    MPM_LAUNCH(L, MPM_K_OTHER, k_grid_mass_adj<T>, blocks_for(c.n_particles, 128), 128, c, st, L.pscene, ggm, gst);
  return cudaGetLastError();
}

template <typename T>
cudaError_t launch_density_l1(const LaunchCtx& L, const T* gm, const T* tgt, double weight, double* loss, T* ggm) {
  const int S = L.p->n_scenes;
  MPM_MEMSET(L, loss, S * sizeof(double));
  int bps = (int)((L.G + 256 * 8 - 1) / (256 * 8));
  if (bps < 1) bps = 1;
  MPM_LAUNCH(L, MPM_K_OTHER, k_density_l1<T>, (unsigned)(S * bps), 256, L.G, gm, tgt, weight, loss, ggm, bps);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// soft contact distance (loss.py:143-162)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_contact_sums(Consts<T> c, const T* __restrict__ st,
                                                      const int* __restrict__ pscene,
                                                      const MpmToolDesc* __restrict__ tools,
                                                      const int* __restrict__ tool_off,
                                                      const double* __restrict__ pose, double* __restrict__ sums) {
  __shared__ StagedTools<T> sh;
  stage_tools(sh, pscene, (int64_t)blockIdx.x * blockDim.x, tools, tool_off, pose);
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = p < c.n_particles;
  const int sc = valid ? pscene[p] : -1;
  const bool per_warp = one_scene(valid, sc);
  const int scene = per_warp ? __shfl_sync(0xffffffffu, sc, 0) : sc;  // -1: a warp past the end
  if (scene < 0) return;
  T x[3] = {T(0), T(0), T(0)};
  if (valid) load_row(st, c.ld, p, 0, 3, x);
  for (int t = tool_off[scene]; t < tool_off[scene + 1]; ++t) {
    if (tools[t].action_dim <= 0) continue;
    double w = 0.0, dw = 0.0;
    if (valid) {
      Tool<T> tl;
      Pose<T> P;
      staged_tool(sh, scene, t, tools, pose, tl, P);
      const T sd = tool_sdf(tl, P, x);
      const double d = (T(0) < sd) ? to_prec<double>(sd) : 0.0;
      w = rcp64(1.0 + d * d * 10000.0);
      dw = d * w;
    }
    if (per_warp) {  // once per warp: a tool's two sums are one address each
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        w += __shfl_xor_sync(0xffffffffu, w, o);
        dw += __shfl_xor_sync(0xffffffffu, dw, o);
      }
      if ((threadIdx.x & 31) != 0) continue;
    }
    atomicAdd(sums + 2 * t, w);
    atomicAdd(sums + 2 * t + 1, dw);
  }
}
__global__ void k_contact_finish(int n_tools, const double* __restrict__ sums, double* __restrict__ min_dist) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n_tools) min_dist[t] = sums[2 * t] > 0 ? sums[2 * t + 1] / sums[2 * t] : 0.0;
}

template <typename T>
cudaError_t launch_soft_contact(const LaunchCtx& L, int n_tools, const T* st, const double* pose, double* sums,
                                double* min_dist) {
  Consts<T> c = make_consts<T>(L);
  MPM_MEMSET(L, sums, 2 * n_tools * sizeof(double));
  if (c.n_particles > 0)
    MPM_LAUNCH(L, MPM_K_OTHER, k_contact_sums<T>, blocks_for(c.n_particles, 128), 128, c, st, L.pscene, L.tools,
               L.tool_off, pose, sums);
  MPM_LAUNCH(L, MPM_K_OTHER, k_contact_finish, blocks_for(n_tools, 64), 64, n_tools, sums, min_dist);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// per-particle tool distances (function.py:79-89)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(128) k_tool_distance(Consts<T> c, const T* __restrict__ st,
                                                       const int* __restrict__ pscene,
                                                       const MpmToolDesc* __restrict__ tools,
                                                       const int* __restrict__ tool_off,
                                                       const int* __restrict__ col_off,
                                                       const double* __restrict__ pose, T* __restrict__ out) {
  int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= c.n_particles) return;
  int sc = pscene[p];
  T x[3];
  load_row(st, c.ld, p, 0, 3, x);
  for (int t = tool_off[sc]; t < tool_off[sc + 1]; ++t) {
    Tool<T> tl;
    Pose<T> P;
    to_tool(tools[t], tl);
    to_pose(pose + 8 * t, P);
    const int col = col_off[t];
    if (fingered(tl.type)) {
      T fa[3], fb[3];
      finger_pos(P, T(-1), fa);
      finger_pos(P, T(1), fb);
      out[(int64_t)col * c.ld + p] = shape_sdf(tl, fa, P.rot, T(0), x);
      out[(int64_t)(col + 1) * c.ld + p] = shape_sdf(tl, fb, P.rot, T(0), x);
    } else {
      out[(int64_t)col * c.ld + p] = tool_sdf(tl, P, x);
    }
  }
}

template <typename T>
cudaError_t launch_tool_distance(const LaunchCtx& L, const int* col_off, int n_cols, const T* st, const double* pose,
                                 T* out) {
  Consts<T> c = make_consts<T>(L);
  MPM_MEMSET(L, out, (int64_t)n_cols * c.ld * sizeof(T));
  if (c.n_particles > 0)
    MPM_LAUNCH(L, MPM_K_OTHER, k_tool_distance<T>, blocks_for(c.n_particles, 128), 128, c, st, L.pscene, L.tools,
               L.tool_off, col_off, pose, out);
  return cudaGetLastError();
}
template cudaError_t launch_tool_distance<float>(const LaunchCtx&, const int*, int, const float*, const double*,
                                                 float*);
template cudaError_t launch_tool_distance<double>(const LaunchCtx&, const int*, int, const double*, const double*,
                                                  double*);

#define MPM_INST_FWD(T, S)                                                                             \
  template cudaError_t launch_substep_fwd<T, S>(const LaunchCtx&, const T*, T*, const double*, const double*, \
                                                const MpmGridStore*, int);
MPM_INST_FWD(float, float)
MPM_INST_FWD(float, double)
MPM_INST_FWD(double, double)
#define MPM_INST_T(T)                                                                                  \
  template cudaError_t launch_grid_mass<T>(const LaunchCtx&, const T*, T*);                            \
  template cudaError_t launch_grid_mass_bwd<T>(const LaunchCtx&, const T*, const T*, T*);              \
  template cudaError_t launch_density_l1<T>(const LaunchCtx&, const T*, const T*, double, double*, T*); \
  template cudaError_t launch_soft_contact<T>(const LaunchCtx&, int, const T*, const double*, double*, double*);
MPM_INST_T(float)
MPM_INST_T(double)

}  // namespace mpm
