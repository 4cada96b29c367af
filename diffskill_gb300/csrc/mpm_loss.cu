// Loss kernels of plb/engine/losses/loss.py beyond the density L1 term:
//   - target-SDF propagation: update_target_sdf / update_target (loss.py:105-134);
//   - SDF loss: compute_sdf_loss_kernel (loss.py:178-180);
//   - IoU: iou_kernel (loss.py:294-308);
//   - hard contact distance: compute_contact_distance_kernel (loss.py:151-155),
//     started from 100000 as compute_loss_kernel does (loss.py:243-244), with an adjoint.
// Dense grids here are real[n_scenes][n_grid^3], node (i,j,k) at (i*n+j)*n+k,
// the C order of the reference's (n,n,n) fields.
#include <climits>

#include "mpm_kernels.cuh"
#include "mpm_launch.h"

namespace mpm {

template <typename T>
Consts<T> make_consts(const LaunchCtx& L);  // mpm_fwd.cu

static inline unsigned blocks_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// products and sums without FMA contraction, so the device rounds every
// operation as the oracle does
MPM_DI float mul_rn(float a, float b) { return __fmul_rn(a, b); }
MPM_DI double mul_rn(double a, double b) { return __dmul_rn(a, b); }
MPM_DI float add_rn(float a, float b) { return __fadd_rn(a, b); }
MPM_DI double add_rn(double a, double b) { return __dadd_rn(a, b); }

// ---------------------------------------------------------------------------
// target SDF: all Jacobi iterations of update_target_sdf in one launch
// ---------------------------------------------------------------------------
// A node whose target density exceeds 1e-4 gets sdf 0 and itself as nearest
// point.  Any other node takes, over the offsets (-3..2)^3 \ {0} in the
// reference's ndrange order, the first strict minimum of
// sqrt(|grid_pos - nearest_copy[v]|^2 + 1e-8) among in-grid neighbours with
// sdf_copy[v] < 1000, else sdf 1000.  A CTA of 128 threads computes patches of
// 4 x 4 x 8 nodes of one scene from a 9 x 9 x 13 shared-memory copy of the
// nearest points around each.  The copy holds a NaN for a neighbour with
// sdf_copy >= 1000, whose squared distance then compares below nothing; a
// candidate is one 16-byte load in FP32.
//
// A candidate replaces the best one iff its rounded distance is smaller.  With
// e = dd + 1e-8, e below the best one's by more than 8 ulp is certainly smaller
// after the square root, and e not below it never is, so the loop compares e and
// keeps the position of the best, without a branch or a square root per
// candidate.  In between (neither on a grid of a power of two, where all dd are
// exact and 1e-5 apart) the node is redone candidate by candidate.  With a branch
// at each candidate whose dd was below the best one's, some lane of a warp took
// it nearly every time: 60 us for a patch, however few were active.
//
// The iterations are separated by a grid barrier of a cooperative launch (all
// CTAs are resident; the wait is bounded, and gives up with
// MPM_STATUS_TIMEOUT).  Two facts leave work out without changing a value:
// - a warp (one plane of a patch) none of whose nodes' 6^3 neighbourhoods changed
//   in the iteration before reproduces its values, which both buffers already
//   hold, so it is skipped, and its patch if all four warps are
//   (changed[t & 1][patch][warp], one bit per node).  The front and what still
//   moves behind it are about a quarter of the warps;
// - once an iteration changes nothing anywhere, neither does any later one
//   (any[3]: iteration t sets any[t % 3], CTA 0 clears any[(t + 1) % 3]).
// What is left sits in a shell that no fixed assignment spreads evenly (with one
// 8^3 tile per CTA an iteration took 50 us, the time of the SM with the most
// active tiles), so the CTAs take the next patch from a counter (next[3], cleared
// like any[3]).  64^3, 128 iterations: 128 launches of one iteration each took
// 1,205 us; now 430.
constexpr int TS_THREADS = 128;
constexpr int TS_A = 4, TS_B = 4, TS_C = 8;             // nodes of a patch
constexpr int TS_HA = 9, TS_HB = 9, TS_HC = 13;         // with the halo of 3 below and 2 above
constexpr int TS_N = TS_HA * TS_HB * TS_HC;
constexpr double TS_INF = 1000.0;

template <typename T>
struct alignas(4 * sizeof(T)) Near {
  T x, y, z, w;
};

// squared distance of p and a nearest point, each operation rounded on its own
template <typename T>
MPM_DI T near_dd(const T* p, const Near<T>& q) {
  const T d0 = p[0] - q.x, d1 = p[1] - q.y, d2 = p[2] - q.z;
  return add_rn(add_rn(mul_rn(d0, d0), mul_rn(d1, d1)), mul_rn(d2, d2));
}

// arrival counter of the grid barrier: barrier k is passed once it reaches
// gridDim.x * (k + 1).  False when the wait ran out.
MPM_DI bool grid_barrier(unsigned* bar, unsigned target, unsigned* status) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    ok = 0;
    for (int poll = 0; poll < (1 << 22); ++poll) {
      unsigned v;
      asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v >= target) {
        ok = 1;
        break;
      }
      __nanosleep(100);
    }
    if (!ok) atomicOr(status, MPM_STATUS_TIMEOUT);
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

template <typename T>
__global__ void __launch_bounds__(TS_THREADS, sizeof(T) == 4 ? 4 : 1) k_target_sdf(int n, int64_t G, int n_scenes, const T* __restrict__ dens,
                                                           T* sdf, T* near, T* w_sdf, T* w_near, double dx, int n_iters,
                                                           int* any, int* next, unsigned* bar, unsigned* changed,
                                                           unsigned* status) {
  __shared__ Near<T> s_near[TS_N];
  __shared__ int s_patch;
  const int na = (n + TS_A - 1) / TS_A, nb = (n + TS_B - 1) / TS_B, nc = (n + TS_C - 1) / TS_C;
  const int per_scene = na * nb * nc, n_patches = n_scenes * per_scene;
  const T inf = T(TS_INF);
  const T none = T(NAN);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l0 = warp, l1 = lane >> 3, l2 = lane & 7;
  for (int iter = 0; iter < n_iters; ++iter) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      any[(iter + 1) % 3] = 0;
      next[(iter + 1) % 3] = 0;
    }
    // the last iteration writes the caller's arrays
    const bool to_out = ((n_iters - 1 - iter) & 1) == 0;
    const T* sdf_c = to_out ? w_sdf : sdf;
    const T* near_c = to_out ? w_near : near;
    T* sdf_o = to_out ? sdf : w_sdf;
    T* near_o = to_out ? near : w_near;
    const unsigned* before = changed + (int64_t)((iter + 1) & 1) * n_patches * 4;
    unsigned* now = changed + (int64_t)(iter & 1) * n_patches * 4;
    while (true) {
      // taken only now: a CTA that held its next patch while it worked on one
      // would make the iteration wait for both
      if (threadIdx.x == 0) s_patch = atomicAdd(next + iter % 3, 1);
      __syncthreads();
      const int patch = s_patch;
      if (patch >= n_patches) break;
      const int scene = patch / per_scene, q0 = patch - scene * per_scene;
      const int pa = q0 / (nb * nc), pb = (q0 / nc) % nb, pc = q0 % nc;
      bool work = true;
      if (iter > 0) {
        // the words of planes l0 - 3 .. l0 + 2 in the patches one before, here
        // and one after along the other axes, less the nodes more than 3 before
        // or 2 after this warp's
        unsigned c = 0u;
        for (int w = lane; w < 54; w += 32) {
          const int plane = pa * TS_A + l0 - 3 + w / 9, db = (w / 3) % 3 - 1, dc = w % 3 - 1;
          const int j = pb + db, k = pc + dc;
          if (plane < 0 || plane >= na * TS_A || j < 0 || j >= nb || k < 0 || k >= nc) continue;
          const unsigned rows = db < 0 ? 0xffffff00u : (db > 0 ? 0x0000ffffu : 0xffffffffu);
          const unsigned cols = dc < 0 ? 0xe0e0e0e0u : (dc > 0 ? 0x03030303u : 0xffffffffu);
          const int at = scene * per_scene + ((plane >> 2) * nb + j) * nc + k;
          c |= __ldcg(before + (int64_t)at * 4 + (plane & 3)) & rows & cols;
        }
        work = __any_sync(0xffffffffu, c != 0u);
        if (!__syncthreads_or(work)) {  // (every thread has read s_patch)
          if (threadIdx.x < 4) now[(int64_t)patch * 4 + threadIdx.x] = 0u;
          continue;
        }
      }
      const int o0 = pa * TS_A, o1 = pb * TS_B, o2 = pc * TS_C;
      const int64_t base = (int64_t)scene * G;
      if (iter > 0) {
        // all of a thread's loads are issued together
        constexpr int kRounds = (TS_N + TS_THREADS - 1) / TS_THREADS;
        T v[kRounds], q[kRounds][3];
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
          const int s = threadIdx.x + TS_THREADS * r;
          const int a = o0 - 3 + s / (TS_HB * TS_HC), b = o1 - 3 + (s / TS_HC) % TS_HB, c = o2 - 3 + s % TS_HC;
          v[r] = inf;
          if (s < TS_N && a >= 0 && a < n && b >= 0 && b < n && c >= 0 && c < n) {
            const int64_t id = base + ((int64_t)a * n + b) * n + c;
            v[r] = __ldcg(sdf_c + id);
#pragma unroll
            for (int k = 0; k < 3; ++k) q[r][k] = __ldcg(near_c + 3 * id + k);
          }
        }
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
          const int s = threadIdx.x + TS_THREADS * r;
          if (s < TS_N)
            s_near[s] = v[r] < inf ? Near<T>{q[r][0], q[r][1], q[r][2], T(0)} : Near<T>{none, none, none, T(0)};
        }
        __syncthreads();
      }
      const int i0 = o0 + l0, i1 = o1 + l1, i2 = o2 + l2;
      bool diff = false;
      if (work && i0 < n && i1 < n && i2 < n) {
        const int64_t id = base + ((int64_t)i0 * n + i1) * n + i2;
        const T gp[3] = {T(double(i0) * dx), T(double(i1) * dx), T(double(i2) * dx)};
        T best = inf, bn[3] = {T(0), T(0), T(0)};
        if (double(dens[id]) > 1e-4) {
          best = T(0);
          bn[0] = gp[0];
          bn[1] = gp[1];
          bn[2] = gp[2];
        } else if (iter > 0) {
          const T keep = T(1) - (sizeof(T) == 4 ? T(4.76837158e-7) : T(1.7763568394002505e-15));  // 1 - 8 ulp
          // three chains over two planes of neighbours each, joined in order: a
          // single chain leaves the few warps of an SM waiting on it
          constexpr int kChains = 3;
          T e_best[kChains], lim[kChains];
          int pos[kChains];
          bool unsure = false;
#pragma unroll
          for (int h = 0; h < kChains; ++h) {
            e_best[h] = T(TS_INF * TS_INF);
            lim[h] = e_best[h] * keep;
            pos[h] = -1;
          }
#pragma unroll 1
          for (int a = 0; a < 2; ++a)
#pragma unroll 1
            for (int b = 0; b < 6; ++b)
#pragma unroll
              for (int c = 0; c < 6; ++c)
#pragma unroll
                for (int h = 0; h < kChains; ++h) {
                  if (h == 1 && c == 3 && a == 1 && b == 3) continue;  // the node itself
                  const int s = ((l0 + 2 * h + a) * TS_HB + (l1 + b)) * TS_HC + l2 + c;
                  const T e = add_rn(near_dd(gp, s_near[s]), T(1e-8));
                  const bool less = e < e_best[h], win = e < lim[h];
                  unsure = unsure || (less && !win);
                  e_best[h] = win ? e : e_best[h];
                  pos[h] = win ? s : pos[h];
                  lim[h] = win ? e * keep : lim[h];
                }
          int at = pos[0];
#pragma unroll
          for (int h = 1; h < kChains; ++h) {
            const bool less = e_best[h] < e_best[0], win = e_best[h] < lim[0];
            unsure = unsure || (less && !win);
            e_best[0] = win ? e_best[h] : e_best[0];
            lim[0] = win ? lim[h] : lim[0];
            at = win ? pos[h] : at;
          }
          if (unsure) {
            at = -1;
            T bdd = T(1e30);
            for (int k = 0; k < 216; ++k) {
              if (k == 3 * 36 + 3 * 6 + 3) continue;
              const int s = ((l0 + k / 36) * TS_HB + (l1 + (k / 6) % 6)) * TS_HC + l2 + k % 6;
              const T dd = near_dd(gp, s_near[s]);
              if (dd < bdd) {
                const T dist = sqrt(add_rn(dd, T(1e-8)));
                if (dist < best) {
                  best = dist;
                  bdd = dd;
                  at = s;
                }
              }
            }
          }
          if (at >= 0) {
            const Near<T> q = s_near[at];
            best = sqrt(add_rn(near_dd(gp, q), T(1e-8)));
            bn[0] = q.x;
            bn[1] = q.y;
            bn[2] = q.z;
          }
        }
        if (iter == 0) {  // both buffers hold iteration 0
          diff = best < inf;
          sdf[id] = w_sdf[id] = best;
          for (int k = 0; k < 3; ++k) near[3 * id + k] = w_near[3 * id + k] = bn[k];
        } else {
          diff = !(best == __ldcg(sdf_c + id)) ||
                 !(bn[0] == __ldcg(near_c + 3 * id) && bn[1] == __ldcg(near_c + 3 * id + 1) &&
                   bn[2] == __ldcg(near_c + 3 * id + 2));
          sdf_o[id] = best;
          near_o[3 * id] = bn[0];
          near_o[3 * id + 1] = bn[1];
          near_o[3 * id + 2] = bn[2];
        }
      }
      const unsigned bits = __ballot_sync(0xffffffffu, diff);
      if (lane == 0) {
        now[(int64_t)patch * 4 + warp] = bits;
        if (bits) any[iter % 3] = 1;
      }
      __syncthreads();  // s_patch and s_near are free
    }
    if (!grid_barrier(bar, gridDim.x * (unsigned)(iter + 1), status)) return;
    if (__ldcg(any + iter % 3) == 0) return;  // uniform over the grid
  }
}

size_t target_sdf_flag_bytes(int n_scenes, int n_grid) {
  auto up = [](int a, int b) { return (int64_t)((a + b - 1) / b); };
  return (size_t)(2 * n_scenes * up(n_grid, TS_A) * up(n_grid, TS_B) * up(n_grid, TS_C)) * 4 * sizeof(unsigned);
}

template <typename T>
cudaError_t launch_target_sdf(const LaunchCtx& L, int* flags, unsigned* changed, const T* dens, T* sdf, T* near,
                              T* work, int n_iters) {
  int n = L.p->n_grid, S = L.p->n_scenes;
  if (n_iters <= 0 || S <= 0) return cudaSuccess;
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_target_sdf<T>, TS_THREADS, 0);
  if (e != cudaSuccess) return e;
  // few enough CTAs that each takes several patches, enough to hide a patch's loads
  if (per_sm > 4) per_sm = 4;
  const int64_t patches = (int64_t)(target_sdf_flag_bytes(S, n) / (8 * sizeof(unsigned)));
  const int64_t resident = (int64_t)per_sm * L.sm_count;
  const unsigned grid = (unsigned)(patches < resident ? patches : resident);
  // each on lines of its own: the waiting CTAs poll bar
  MPM_MEMSET(L, flags, kTargetSdfFlags * sizeof(int));
  int *any = flags, *next = flags + 64;
  unsigned* bar = reinterpret_cast<unsigned*>(flags + 128);
  int64_t G = L.G;
  T* w_near = work + (int64_t)S * G;
  double dx = L.p->dx;
  unsigned* status = L.status;
  void* args[] = {&n,  &G,       &S,   (void*)&dens, &sdf, &near,    &work,  &w_near,
                  &dx, &n_iters, &any, &next,        &bar, &changed, &status};
  const int slot = prof_begin(L.prof, L.stream);
  e = cudaLaunchCooperativeKernel((const void*)k_target_sdf<T>, dim3(grid), dim3(TS_THREADS), args, 0, L.stream);
  prof_end(L.prof, slot, MPM_K_OTHER, L.stream);
  ++*L.launches;
  return e != cudaSuccess ? e : cudaGetLastError();
}

// ---------------------------------------------------------------------------
// SDF loss and IoU: one thread-block cluster per scene, fixed-order FP64
// reductions (each thread its elements in order, lanes, warps, then the
// cluster's CTAs through distributed shared memory; no scratch in global
// memory, so calls on several streams stay independent).
//
// A node where both factors are zero adds nothing, and most of a grid is empty:
// a warp whose 32 nodes are all empty skips the FP64 additions (an SM issues one
// every 16 cycles).  With one CTA per scene and no such test the FP64 pipe of a
// single SM did all the work: 64^3 IoU 525 us, SDF loss 151 us now 24 and 15.
// ---------------------------------------------------------------------------
constexpr int RED_THREADS = 512;
// 16 CTAs per scene while they are few (a non-portable size), else 8
inline int reduction_cluster(int n_scenes) { return n_scenes <= 8 ? 16 : 8; }

MPM_DI unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
MPM_DI unsigned cluster_size() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// (.aligned: the warp's threads execute it together, so those that come from a branch
// meet first)
MPM_DI void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// v of CTA `rank`'s shared variable at the address of `mine`
MPM_DI double cluster_read(const double* mine, unsigned rank) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(mine);
  unsigned b;
  double v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(b) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(b) : "memory");
  return v;
}
MPM_DI double op_of(double a, double b, bool max) { return max ? fmax(a, b) : a + b; }
// Reduces N values over a cluster: values below NMAX by fmax, the others by
// addition.  The result is in v of thread 0 of CTA 0.
template <int N, int NMAX>
MPM_DI void cluster_reduce(double (&v)[N]) {
  __shared__ double warp_part[N][RED_THREADS / 32], part[N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[k] = op_of(v[k], __shfl_xor_sync(0xffffffffu, v[k], o), k < NMAX);
    if ((threadIdx.x & 31) == 0) warp_part[k][threadIdx.x >> 5] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < N) {
    const int k = threadIdx.x;
    double s = warp_part[k][0];
    for (int w = 1; w < RED_THREADS / 32; ++w) s = op_of(s, warp_part[k][w], k < NMAX);
    part[k] = s;
  }
  cluster_sync();
  if (cluster_rank() == 0 && threadIdx.x == 0) {
    const unsigned n = cluster_size();
#pragma unroll
    for (int k = 0; k < N; ++k) {
      double s = part[k];
      for (unsigned r = 1; r < n; ++r) s = op_of(s, cluster_read(part + k, r), k < NMAX);
      v[k] = s;
    }
  }
  cluster_sync();  // no CTA leaves while its partial sums are read
}

// loss[s] = weight * sum_I sdf*m; g_grid_m += weight * sdf
template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_sdf_loss(int64_t G, const T* __restrict__ gm,
                                                          const T* __restrict__ sdf, double weight,
                                                          double* __restrict__ loss, T* __restrict__ ggm) {
  const unsigned n = cluster_size(), rank = cluster_rank();
  const int scene = (int)(blockIdx.x / n);
  const int64_t base = (int64_t)scene * G;
  double acc[1] = {0.0};
  for (int64_t i0 = (int64_t)rank * RED_THREADS; i0 < G; i0 += (int64_t)n * RED_THREADS) {
    const int64_t i = i0 + threadIdx.x;
    T term = T(0);
    if (i < G) {
      const T sd = sdf[base + i];
      term = sd * gm[base + i];
      if (ggm) ggm[base + i] += T(weight) * sd;
    }
    if (__any_sync(0xffffffffu, term != T(0))) acc[0] += double(term);
  }
  cluster_reduce<1, 0>(acc);
  if (rank == 0 && threadIdx.x == 0) loss[scene] = weight * acc[0];
}

template <typename T>
__global__ void __launch_bounds__(RED_THREADS) k_iou(int64_t G, const T* __restrict__ gm, const T* __restrict__ tgt,
                                                     double* __restrict__ iou) {
  const unsigned n = cluster_size(), rank = cluster_rank();
  const int scene = (int)(blockIdx.x / n);
  const int64_t base = (int64_t)scene * G;
  // the maxima start at 0 as the reference's atomic_max accumulators do
  T ma = T(0), mb = T(0);
  double I = 0.0, Ua = 0.0, Ub = 0.0;
  for (int64_t i0 = (int64_t)rank * RED_THREADS; i0 < G; i0 += (int64_t)n * RED_THREADS) {
    const int64_t i = i0 + threadIdx.x;
    const T a = i < G ? gm[base + i] : T(0), b = i < G ? tgt[base + i] : T(0);
    if (__any_sync(0xffffffffu, a != T(0) || b != T(0))) {
      const double da = double(a), db = double(b);
      ma = fmax(ma, a);
      mb = fmax(mb, b);
      I += da * db;
      Ua += da;
      Ub += db;
    }
  }
  double v[5] = {double(ma), double(mb), I, Ua, Ub};
  cluster_reduce<5, 2>(v);
  if (rank == 0 && threadIdx.x == 0) {
    const double In = v[2] / v[0] / v[1];
    const double U = v[3] / v[0] + v[4] / v[1];
    iou[scene] = In / (U - In);
  }
}

// one cluster of `reduction_cluster` CTAs per scene
template <typename... KArgs, typename... Args>
static cudaError_t launch_reduction(const LaunchCtx& L, void (*kernel)(KArgs...), Args... args) {
  const int S = L.p->n_scenes, size = reduction_cluster(S);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(S * size));
  cfg.blockDim = dim3(RED_THREADS);
  cfg.stream = L.stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)size;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int slot = prof_begin(L.prof, L.stream);
  e = cudaLaunchKernelEx(&cfg, kernel, args...);
  prof_end(L.prof, slot, MPM_K_OTHER, L.stream);
  ++*L.launches;
  return e;
}

template <typename T>
cudaError_t launch_sdf_loss(const LaunchCtx& L, const T* gm, const T* sdf, double weight, double* loss, T* ggm) {
  return L.p->n_scenes > 0 ? launch_reduction(L, k_sdf_loss<T>, L.G, gm, sdf, weight, loss, ggm) : cudaSuccess;
}
template <typename T>
cudaError_t launch_iou(const LaunchCtx& L, const T* gm, const T* tgt, double* iou) {
  return L.p->n_scenes > 0 ? launch_reduction(L, k_iou<T>, L.G, gm, tgt, iou) : cudaSuccess;
}

// ---------------------------------------------------------------------------
// hard contact distance: min over particles of max(sdf, 0) per movable tool
// ---------------------------------------------------------------------------
// The minimum is an atomicMin on the bit pattern of the non-negative FP64
// distance (which orders like the value), kept in min_dist itself; a second
// pass takes the lowest particle index attaining it.
template <typename T>
MPM_DI double contact_d(const Tool<T>& tl, const Pose<T>& P, const T* x) {
  const T sd = tool_sdf(tl, P, x);
  return (T(0) < sd) ? double(sd) : 0.0;
}

__global__ void k_contact_min_init(int n_tools, double* __restrict__ min_dist, int64_t* __restrict__ argmin) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tools) return;
  min_dist[t] = 100000.0;
  argmin[t] = -1;  // all bits set: the largest value for the unsigned atomicMin
}

template <typename T>
__global__ void __launch_bounds__(128) k_contact_min(Consts<T> c, const T* __restrict__ st,
                                                     const int* __restrict__ pscene,
                                                     const MpmToolDesc* __restrict__ tools,
                                                     const int* __restrict__ tool_off,
                                                     const double* __restrict__ pose, double* __restrict__ min_dist) {
  __shared__ StagedTools<T> sh;
  stage_tools(sh, pscene, (int64_t)blockIdx.x * blockDim.x, tools, tool_off, pose);
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = p < c.n_particles;
  const int sc = valid ? pscene[p] : -1;
  const bool per_warp = one_scene(valid, sc);
  const int scene = per_warp ? __shfl_sync(0xffffffffu, sc, 0) : sc;
  if (scene < 0) return;
  T x[3] = {T(0), T(0), T(0)};
  if (valid) load_row(st, c.ld, p, 0, 3, x);
  for (int t = tool_off[scene]; t < tool_off[scene + 1]; ++t) {
    if (tools[t].action_dim <= 0) continue;
    unsigned long long d = ~0ull;  // the bits of a non-negative distance order like it
    if (valid) {
      Tool<T> tl;
      Pose<T> P;
      staged_tool(sh, scene, t, tools, pose, tl, P);
      d = (unsigned long long)__double_as_longlong(contact_d(tl, P, x));
    }
    if (per_warp) {  // one atomic per warp
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long e = __shfl_xor_sync(0xffffffffu, d, o);
        d = e < d ? e : d;
      }
      if ((threadIdx.x & 31) != 0) continue;
    }
    atomicMin(reinterpret_cast<unsigned long long*>(min_dist + t), d);
  }
}

template <typename T>
__global__ void __launch_bounds__(128) k_contact_argmin(Consts<T> c, const T* __restrict__ st,
                                                        const int* __restrict__ pscene,
                                                        const MpmToolDesc* __restrict__ tools,
                                                        const int* __restrict__ tool_off,
                                                        const double* __restrict__ pose,
                                                        const double* __restrict__ min_dist,
                                                        int64_t* __restrict__ argmin) {
  __shared__ StagedTools<T> sh;
  stage_tools(sh, pscene, (int64_t)blockIdx.x * blockDim.x, tools, tool_off, pose);
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= c.n_particles) return;
  const int sc = pscene[p];
  T x[3];
  load_row(st, c.ld, p, 0, 3, x);
  for (int t = tool_off[sc]; t < tool_off[sc + 1]; ++t) {
    if (tools[t].action_dim <= 0) continue;
    Tool<T> tl;
    Pose<T> P;
    staged_tool(sh, sc, t, tools, pose, tl, P);
    const double d = contact_d(tl, P, x);
    if (d == min_dist[t]) atomicMin(reinterpret_cast<unsigned long long*>(argmin + t), (unsigned long long)p);
  }
}

__global__ void k_contact_min_finish(const MpmToolDesc* __restrict__ tools, int n_tools,
                                     double* __restrict__ min_dist) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n_tools && tools[t].action_dim <= 0) min_dist[t] = 0.0;
}

template <typename T>
cudaError_t launch_contact_min(const LaunchCtx& L, int n_tools, const T* st, const double* pose, double* min_dist,
                               int64_t* argmin) {
  Consts<T> c = make_consts<T>(L);
  MPM_LAUNCH(L, MPM_K_OTHER, k_contact_min_init, blocks_for(n_tools, 64), 64, n_tools, min_dist, argmin);
  if (c.n_particles > 0) {
    MPM_LAUNCH(L, MPM_K_OTHER, k_contact_min<T>, blocks_for(c.n_particles, 128), 128, c, st, L.pscene, L.tools,
               L.tool_off, pose, min_dist);
    MPM_LAUNCH(L, MPM_K_OTHER, k_contact_argmin<T>, blocks_for(c.n_particles, 128), 128, c, st, L.pscene, L.tools,
               L.tool_off, pose, min_dist, argmin);
  }
  MPM_LAUNCH(L, MPM_K_OTHER, k_contact_min_finish, blocks_for(n_tools, 64), 64, L.tools, n_tools, min_dist);
  return cudaGetLastError();
}

// adjoint: d min / d x_argmin = d max(sdf,0) / dx, zero when sdf <= 0
template <typename T>
__global__ void k_contact_min_adj(Consts<T> c, const T* __restrict__ st, const MpmToolDesc* __restrict__ tools,
                                  int n_tools, const double* __restrict__ pose, const int64_t* __restrict__ argmin,
                                  const double* __restrict__ g_min, T* __restrict__ gst,
                                  double* __restrict__ g_pose) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tools) return;
  const int64_t p = argmin[t];
  if (tools[t].action_dim <= 0 || p < 0 || p >= c.n_particles || g_min[t] == 0.0) return;
  T x[3];
  load_row(st, c.ld, p, 0, 3, x);
  Tool<T> tl;
  Pose<T> P;
  to_tool(tools[t], tl);
  to_pose(pose + 8 * t, P);
  if (!(T(0) < tool_sdf(tl, P, x))) return;
  T gx[3] = {T(0), T(0), T(0)};
  PoseGrad<T> gP;
  gP.zero();
  tool_sdf_vjp(tl, P, x, T(g_min[t]), gx, gP);
  for (int k = 0; k < 3; ++k) atomicAdd(gst + (int64_t)k * c.ld + p, gx[k]);
  for (int k = 0; k < 3; ++k) g_pose[8 * t + k] += double(gP.pos[k]);
  for (int k = 0; k < 4; ++k) g_pose[8 * t + 3 + k] += double(gP.rot[k]);
  g_pose[8 * t + 7] += double(gP.gap);
}

template <typename T>
cudaError_t launch_contact_min_bwd(const LaunchCtx& L, int n_tools, const T* st, const double* pose,
                                   const int64_t* argmin, const double* g_min, T* gst, double* g_pose) {
  Consts<T> c = make_consts<T>(L);
  MPM_LAUNCH(L, MPM_K_OTHER, k_contact_min_adj<T>, blocks_for(n_tools, 64), 64, c, st, L.tools, n_tools, pose,
             argmin, g_min, gst, g_pose);
  return cudaGetLastError();
}

#define MPM_INST_LOSS(T)                                                                                       \
  template cudaError_t launch_target_sdf<T>(const LaunchCtx&, int*, unsigned*, const T*, T*, T*, T*, int); \
  template cudaError_t launch_sdf_loss<T>(const LaunchCtx&, const T*, const T*, double, double*, T*);          \
  template cudaError_t launch_iou<T>(const LaunchCtx&, const T*, const T*, double*);                          \
  template cudaError_t launch_contact_min<T>(const LaunchCtx&, int, const T*, const double*, double*, int64_t*); \
  template cudaError_t launch_contact_min_bwd<T>(const LaunchCtx&, int, const T*, const double*, const int64_t*, \
                                                 const double*, T*, double*);
MPM_INST_LOSS(float)
MPM_INST_LOSS(double)

}  // namespace mpm
