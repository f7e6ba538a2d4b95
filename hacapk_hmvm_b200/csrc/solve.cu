// Krylov solvers on a resident plan: the callers of the HMVM.
//
// BiCGSTAB restates HACApK_bicgstab_lfmtx (src_lhdump/m_HACApK_solve.f90:
// 977-1028), van der Vorst's BiCGSTAB with the shadow residual r0 = b - A u0:
// per step two H-matrix products (hmvm_b200_apply on the device-resident
// matrix) and five inner products.  GCR(m) restates HACApK_gcrm_lfmtx
// (m_HACApK_solve.f90:1277-1342): one product per step, search directions
// A-orthogonalised against the last m (restarted cyclically).  All vectors
// stay on the device; the inner products are summed in a fixed order
// (per-block partial sums, then one block), so a solve is repeatable bit for
// bit.  BiCGSTAB's scalars stay on the device too: every kernel that needs one
// adds up the partial sums itself, and the host reads one record per step, for
// the stopping test ||r|| / ||b|| < eps.  GCR(m) reads its inner products back.
//
// BiCGSTAB at N = 12,000 (FP64, 7 steps, 15 products of 45 us): 2.1 ms with work
// vectors allocated and freed by each call (more where the allocator is slow) and
// three round trips to the host per step, 0.70 to 0.86 ms with the plan's workspace
// and one.  What is left is the products and the gaps before them.
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <vector>

#include "hmvm_b200.h"

namespace hmvm {
int set_error(int status, const std::string& msg);
// Device memory of a plan for the length of a solve (hmvm_b200.cu).
int solve_workspace(hmvm_plan* plan, size_t bytes, void** dev, bool* kept);
}
using hmvm::set_error;

namespace {

constexpr int kDotBlocks = 256;
constexpr int kDotThreads = 256;

// part[b * 2 + j] = sum over the block's strided elements of x_j . y_j
template <typename T>
__global__ void dot2_partial(const T* __restrict__ x0, const T* __restrict__ y0, const T* __restrict__ x1,
                             const T* __restrict__ y1, int n, double* __restrict__ part) {
  __shared__ double s0[kDotThreads], s1[kDotThreads];
  double a0 = 0.0, a1 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    a0 += (double)x0[i] * (double)y0[i];
    if (x1) a1 += (double)x1[i] * (double)y1[i];
  }
  s0[threadIdx.x] = a0;
  s1[threadIdx.x] = a1;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      s0[threadIdx.x] += s0[threadIdx.x + w];
      s1[threadIdx.x] += s1[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s0[0];
    part[2 * blockIdx.x + 1] = s1[0];
  }
}
__global__ void dot2_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double s0[kDotBlocks], s1[kDotBlocks];
  const int t = threadIdx.x;
  s0[t] = t < nb ? part[2 * t] : 0.0;
  s1[t] = t < nb ? part[2 * t + 1] : 0.0;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (t < w) {
      s0[t] += s0[t + w];
      s1[t] += s1[t + w];
    }
    __syncthreads();
  }
  if (t == 0) {
    out[0] = s0[0];
    out[1] = s1[0];
  }
}

// part[(j * kDotBlocks + b)] = block b's partial sum of x_j . y, x_j = x + j * ldx
template <typename T>
__global__ void dotm_partial(const T* __restrict__ x, size_t ldx, const T* __restrict__ y, int n,
                             double* __restrict__ part) {
  __shared__ double s[kDotThreads];
  const T* xj = x + blockIdx.y * ldx;
  double a = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    a += (double)xj[i] * (double)y[i];
  s[threadIdx.x] = a;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) s[threadIdx.x] += s[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.y * gridDim.x + blockIdx.x] = s[0];
}
// out[j] = sum of part[j * nb .. j * nb + nb), one block per j
__global__ void dotm_final(const double* __restrict__ part, int nb, double* __restrict__ out) {
  __shared__ double s[kDotBlocks];
  const int t = threadIdx.x;
  s[t] = t < nb ? part[blockIdx.x * nb + t] : 0.0;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (t < w) s[t] += s[t + w];
    __syncthreads();
  }
  if (t == 0) out[blockIdx.x] = s[0];
}

constexpr int kMaxRestart = 64;
struct Betas {
  double b[kMaxRestart];
};
// GCR direction update, per element in the reference's order
// (m_HACApK_solve.f90:1331-1337): for il = 0..k-1,
//   p_new += beta_il * p_il,  ap_new += beta_il * ap_il,
// where slot `self` is p_new / ap_new itself (the restart step, at which the
// new direction reuses the oldest slot) and reads its current value.
template <typename T>
__global__ void gcr_update(T* __restrict__ p, T* __restrict__ ap, size_t ld, int k, int self, Betas be, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    T* pn = p + (size_t)self * ld;
    T* an = ap + (size_t)self * ld;
    T vp = pn[i], va = an[i];
    for (int il = 0; il < k; il++) {
      const T wp = il == self ? vp : p[il * ld + i];
      const T wa = il == self ? va : ap[il * ld + i];
      vp = (T)((double)vp + be.b[il] * (double)wp);
      va = (T)((double)va + be.b[il] * (double)wa);
    }
    pn[i] = vp;
    an[i] = va;
  }
}

// z = x + a * y + b * w (w may be NULL)
template <typename T>
__global__ void axpbyz(T* __restrict__ z, const T* __restrict__ x, double a, const T* __restrict__ y, double b,
                       const T* __restrict__ w, int n) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double v = (double)x[i] + a * (double)y[i];
    if (w) v += b * (double)w[i];
    z[i] = (T)v;
  }
}

// Launches a kernel and reports a failed launch at once: the workspace outlives a
// solve, so a scalar that a kernel did not write would be an earlier solve's.
template <typename... P, typename... A>
int launch(cudaStream_t st, void (*kernel)(P...), dim3 grid, int threads, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3((unsigned)threads);
  c.stream = st;
  const cudaError_t e = cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
  return e == cudaSuccess ? HMVM_OK : set_error(HMVM_ECUDA, std::string("solver kernel: ") + cudaGetErrorString(e));
}
int copied(cudaError_t e) { return e == cudaSuccess ? HMVM_OK : set_error(HMVM_ECUDA, "solver: vector copy"); }

template <typename T>
struct Solver {
  hmvm_plan* plan;
  int n;
  cudaStream_t st;
  double* part;  // [2 * kDotBlocks + 2]
  double host[2];

  int dot2(const T* x0, const T* y0, const T* x1, const T* y1, double* d0, double* d1) {
    int rc = launch(st, dot2_partial<T>, kDotBlocks, kDotThreads, x0, y0, x1, y1, n, part);
    if (!rc) rc = launch(st, dot2_final, 1, kDotBlocks, part, kDotBlocks, part + 2 * kDotBlocks);
    if (rc) return rc;
    if (cudaMemcpyAsync(host, part + 2 * kDotBlocks, 2 * sizeof(double), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return set_error(HMVM_ECUDA, "bicgstab: inner products");
    *d0 = host[0];
    if (d1) *d1 = host[1];
    return HMVM_OK;
  }
  int lin(T* z, const T* x, double a, const T* y, double b = 0.0, const T* w = nullptr) {
    return launch(st, axpbyz<T>, (n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184, 256, z, x, a, y, b, w, n);
  }
};

// ---- BiCGSTAB ------------------------------------------------------------------
// The record that the host reads once per step, and the scalars between kernels.
struct BicgState {
  double bb, rr;             // b . b and r . r
  double alpha, zeta, beta;  // of the last step
  double nom;                // shadow . r at its start
  int32_t breakdown;         // 1: shadow . A p vanished (the step was not taken)
  int32_t _pad;
};

// The two sums of kDotBlocks partial pairs, in dot2_final's order, for every
// thread of a block of kDotBlocks threads.
__device__ __forceinline__ void sum_partials(const double* __restrict__ part, double& a, double& b) {
  __shared__ double s0[kDotBlocks], s1[kDotBlocks];
  const int t = threadIdx.x;
  s0[t] = part[2 * t];
  s1[t] = part[2 * t + 1];
  __syncthreads();
  for (int w = kDotBlocks / 2; w > 0; w >>= 1) {
    if (t < w) {
      s0[t] += s0[t + w];
      s1[t] += s1[t + w];
    }
    __syncthreads();
  }
  a = s0[0];
  b = s1[0];
}
// The block's sums of every thread's (a, b) into its pair of `part`.
__device__ __forceinline__ void block_partials(double a, double b, double* __restrict__ part) {
  __shared__ double s0[kDotThreads], s1[kDotThreads];
  s0[threadIdx.x] = a;
  s1[threadIdx.x] = b;
  __syncthreads();
  for (int w = kDotThreads / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) {
      s0[threadIdx.x] += s0[threadIdx.x + w];
      s1[threadIdx.x] += s1[threadIdx.x + w];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = s0[0];
    part[2 * blockIdx.x + 1] = s1[0];
  }
}
static_assert(kDotBlocks == kDotThreads, "one thread per partial pair");

// r = shadow = b - A u; partial sums of b . b and r . r
template <typename T>
__global__ void bicg_start(const T* __restrict__ b, const T* __restrict__ au, T* __restrict__ r, T* __restrict__ sh,
                           int n, double* __restrict__ part) {
  double a0 = 0.0, a1 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double bi = (double)b[i];
    const T ri = (T)(bi - (double)au[i]);
    r[i] = ri;
    sh[i] = ri;
    a0 += bi * bi;
    a1 += (double)ri * (double)ri;
  }
  block_partials(a0, a1, part);
}
// The scalars of the step that ended (first: of the start), then
// p = r + beta (p - zeta A p)
template <typename T>
__global__ void bicg_direction(const T* __restrict__ r, const T* __restrict__ akp, T* __restrict__ p, int n, bool first,
                               const double* __restrict__ part, const BicgState* __restrict__ in,
                               BicgState* __restrict__ out) {
  double d0, d1;
  sum_partials(part, d0, d1);
  const BicgState st = first ? BicgState{} : *in;
  const double beta = first ? 0.0 : st.alpha / st.zeta * d0 / st.nom;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    BicgState o = st;
    if (first) o.bb = d0;
    o.rr = d1;
    o.beta = beta;
    *out = o;
  }
  if (st.breakdown) return;
  const double bz = -beta * st.zeta;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    double v = (double)r[i];
    if (!first) {
      v += beta * (double)p[i];
      v += bz * (double)akp[i];
    }
    p[i] = (T)v;
  }
}
// alpha from the partial sums of shadow . r and shadow . A p; t = r - alpha A p
template <typename T>
__global__ void bicg_half(const T* __restrict__ r, const T* __restrict__ akp, T* __restrict__ t, int n,
                          const double* __restrict__ part, BicgState* __restrict__ state) {
  double nom, den;
  sum_partials(part, nom, den);
  const double alpha = den != 0.0 ? nom / den : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    state->nom = nom;
    state->alpha = alpha;
    state->breakdown = den == 0.0;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    t[i] = (T)((double)r[i] + -alpha * (double)akp[i]);
}
// zeta from the partial sums of A t . t and A t . A t; u += alpha p + zeta t,
// r = t - zeta A t; partial sums of shadow . r and r . r.  A broken-down step
// leaves u, r and the sums alone.
template <typename T>
__global__ void bicg_step(T* __restrict__ u, T* __restrict__ r, const T* __restrict__ p, const T* __restrict__ t,
                          const T* __restrict__ akt, const T* __restrict__ sh, int n, const double* __restrict__ part,
                          BicgState* __restrict__ state, double* __restrict__ part_out) {
  double znom, zden;
  sum_partials(part, znom, zden);
  if (state->breakdown) return;
  const double alpha = state->alpha, zeta = zden != 0.0 ? znom / zden : 0.0;
  if (blockIdx.x == 0 && threadIdx.x == 0) state->zeta = zeta;
  double a0 = 0.0, a1 = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const double ti = (double)t[i];
    double v = (double)u[i] + alpha * (double)p[i];
    v += zeta * ti;
    u[i] = (T)v;
    const T ri = (T)(ti + -zeta * (double)akt[i]);
    r[i] = ri;
    a0 += (double)sh[i] * (double)ri;
    a1 += (double)ri * (double)ri;
  }
  block_partials(a0, a1, part_out);
}

template <typename T>
int bicgstab_t(hmvm_plan* plan, int n, const T* b, T* u, int max_steps, double eps, int32_t* steps_out,
               double* relres_out, cudaStream_t st) {
  // r, shadow, p, t, A p, A t; three sets of partial sums; two state records
  const size_t ld = ((size_t)n + 31) / 32 * 32, vec_bytes = 6 * ld * sizeof(T);
  void* ws = nullptr;
  bool kept = false;
  int rc = hmvm::solve_workspace(plan, vec_bytes + 6 * kDotBlocks * sizeof(double) + 2 * sizeof(BicgState), &ws, &kept);
  if (rc) return set_error(HMVM_ENOMEM, "bicgstab: device vectors");
  T *r = static_cast<T*>(ws), *sh = r + ld, *p = r + 2 * ld, *t = r + 3 * ld, *akp = r + 4 * ld, *akt = r + 5 * ld;
  double* part0 = reinterpret_cast<double*>(static_cast<char*>(ws) + vec_bytes);
  double *part1 = part0 + 2 * kDotBlocks, *part2 = part1 + 2 * kDotBlocks;
  BicgState* state = reinterpret_cast<BicgState*>(part2 + 2 * kDotBlocks);  // [2], alternating
  BicgState h{};
  double bnorm = 0, relres = 0;
  int steps = 0;
  rc = hmvm_b200_apply(plan, u, akt, st);
  if (!rc) rc = launch(st, bicg_start<T>, kDotBlocks, kDotThreads, b, akt, r, sh, n, part0);
  for (int k = 0; !rc; k++) {
    // the next direction; its record tells how the step before it ended
    BicgState *in = state + (k & 1 ? 0 : 1), *out = state + (k & 1 ? 1 : 0);
    rc = launch(st, bicg_direction<T>, kDotBlocks, kDotThreads, r, akp, p, n, k == 0, part0, in, out);
    if (rc) break;
    if (cudaMemcpyAsync(&h, out, sizeof h, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      rc = set_error(HMVM_ECUDA, "bicgstab: inner products");
      break;
    }
    if (h.breakdown) {
      rc = set_error(HMVM_EINVAL, "bicgstab: breakdown (shadow residual orthogonal to A p)");
      break;
    }
    if (k == 0) {
      bnorm = std::sqrt(h.bb);
      relres = bnorm > 0 ? std::sqrt(h.rr) / bnorm : 0.0;
    } else {
      steps = k;
      relres = std::sqrt(h.rr) / bnorm;
      if (h.zeta == 0.0 || h.nom == 0.0) {
        rc = set_error(HMVM_EINVAL, "bicgstab: breakdown (zeta or rho vanished)");
        break;
      }
    }
    if (!(relres >= eps) || k >= max_steps) break;
    rc = hmvm_b200_apply(plan, p, akp, st);
    if (!rc) rc = launch(st, dot2_partial<T>, kDotBlocks, kDotThreads, sh, r, sh, akp, n, part1);
    if (!rc) rc = launch(st, bicg_half<T>, kDotBlocks, kDotThreads, r, akp, t, n, part1, out);
    if (!rc) rc = hmvm_b200_apply(plan, t, akt, st);
    if (!rc) rc = launch(st, dot2_partial<T>, kDotBlocks, kDotThreads, akt, t, akt, akt, n, part2);
    if (!rc) rc = launch(st, bicg_step<T>, kDotBlocks, kDotThreads, u, r, p, t, akt, sh, n, part2, out, part0);
  }
  cudaStreamSynchronize(st);
  if (!kept) cudaFree(ws);
  if (steps_out) *steps_out = steps;
  if (relres_out) *relres_out = relres;
  if (!rc) rc = hmvm_b200_plan_status(plan);
  return rc;
}

template <typename T>
int gcrm_t(hmvm_plan* plan, int n, const T* b, T* u, int max_steps, int m, double eps, int32_t* steps_out,
           double* relres_out, cudaStream_t st) {
  // r, ar, then the m directions p and their products ap; partial sums and inner products
  const size_t ld = ((size_t)n + 31) / 32 * 32, vec_bytes = sizeof(T) * ld * (2 + 2 * (size_t)m);
  void* ws = nullptr;
  bool kept = false;
  if (hmvm::solve_workspace(plan, vec_bytes + sizeof(double) * ((size_t)kDotBlocks * (m + 2) + m + 2), &ws, &kept))
    return set_error(HMVM_ENOMEM, "gcrm: device vectors");
  T *r = static_cast<T*>(ws), *ar = r + ld, *p = r + 2 * ld, *ap = r + (2 + (size_t)m) * ld;
  double* part = reinterpret_cast<double*>(static_cast<char*>(ws) + vec_bytes);
  double* dots = part + (size_t)kDotBlocks * (m + 2);
  Solver<T> s{plan, n, st, part, {0, 0}};
  std::vector<double> capap(m, 0.0), hd(m, 0.0);
  int rc = HMVM_OK;
  double bb = 0, rr = 0, relres = 0;
  int steps = 0;
  // r = b - A u; p_0 = r
  rc = hmvm_b200_apply(plan, u, ar, st);
  if (!rc) rc = s.lin(r, b, -1.0, ar);
  if (!rc) rc = copied(cudaMemcpyAsync(p, r, sizeof(T) * n, cudaMemcpyDeviceToDevice, st));
  if (!rc) rc = s.dot2(b, b, r, r, &bb, &rr);
  const double bnorm = std::sqrt(bb);
  relres = bnorm > 0 ? std::sqrt(rr) / bnorm : 0.0;
  if (!rc && relres >= eps && max_steps > 0) rc = hmvm_b200_apply(plan, p, ap, st);  // ap_0 = A p_0
  for (int in = 1; !rc && relres >= eps && in <= max_steps; in++) {
    const int ik = (in - 1) % m;
    T* q = ap + (size_t)ik * ld;
    double nom, qq;
    rc = s.dot2(q, r, q, q, &nom, &qq);
    if (rc) break;
    if (qq == 0.0) {
      rc = set_error(HMVM_EINVAL, "gcrm: breakdown (A p vanished)");
      break;
    }
    capap[ik] = qq;
    const double alpha = nom / qq;
    rc = s.lin(u, u, alpha, p + (size_t)ik * ld);  // u += alpha p_ik
    if (!rc) rc = s.lin(r, r, -alpha, q);          // r -= alpha ap_ik
    if (!rc) rc = s.dot2(r, r, nullptr, nullptr, &rr, nullptr);
    if (rc) break;
    relres = std::sqrt(rr) / bnorm;
    steps = in;
    if (relres < eps || in == max_steps) break;
    rc = hmvm_b200_apply(plan, r, ar, st);  // ar = A r
    const int ikn = in % m;
    if (!rc) rc = copied(cudaMemcpyAsync(p + (size_t)ikn * ld, r, sizeof(T) * n, cudaMemcpyDeviceToDevice, st));
    if (!rc) rc = copied(cudaMemcpyAsync(ap + (size_t)ikn * ld, ar, sizeof(T) * n, cudaMemcpyDeviceToDevice, st));
    // beta_il = -(ap_il . ar) / capap_il for il = 0..ik, all against the same ar
    const int k = ik + 1;
    if (!rc) rc = launch(st, dotm_partial<T>, dim3(kDotBlocks, k), kDotThreads, ap, ld, ar, n, part);
    if (!rc) rc = launch(st, dotm_final, k, kDotBlocks, part, kDotBlocks, dots);
    if (rc) break;
    if (cudaMemcpyAsync(hd.data(), dots, sizeof(double) * k, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess) {
      rc = set_error(HMVM_ECUDA, "gcrm: inner products");
      break;
    }
    Betas be;
    for (int il = 0; il < k; il++) be.b[il] = -hd[il] / capap[il];
    rc = launch(st, gcr_update<T>, (n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184, 256, p, ap, ld, k, ikn, be, n);
  }
  cudaStreamSynchronize(st);
  if (!kept) cudaFree(ws);
  if (steps_out) *steps_out = steps;
  if (relres_out) *relres_out = relres;
  if (!rc) rc = hmvm_b200_plan_status(plan);
  return rc;
}

}  // namespace

extern "C" int hmvm_b200_bicgstab(hmvm_plan* plan, const void* b_dev, void* u_dev, int32_t max_steps, double eps,
                                  int32_t* steps, double* relres, void* stream) {
  hmvm_plan_info info;
  int rc = hmvm_b200_plan_get_info(plan, &info);
  if (rc) return rc;
  if (info.nd > 0 && (!b_dev || !u_dev)) return set_error(HMVM_EINVAL, "b or u is NULL");
  if (max_steps < 0 || !(eps >= 0.0)) return set_error(HMVM_EINVAL, "max_steps < 0 or eps not >= 0");
  if (info.nd == 0) {
    if (steps) *steps = 0;
    if (relres) *relres = 0.0;
    return HMVM_OK;
  }
  int cur = 0;
  cudaGetDevice(&cur);
  if (cudaSetDevice(info.device) != cudaSuccess) return set_error(HMVM_ECUDA, "cannot select the plan's device");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (info.precision == HMVM_FP32)
    rc = bicgstab_t<float>(plan, info.nd, static_cast<const float*>(b_dev), static_cast<float*>(u_dev), max_steps,
                           eps, steps, relres, st);
  else
    rc = bicgstab_t<double>(plan, info.nd, static_cast<const double*>(b_dev), static_cast<double*>(u_dev), max_steps,
                            eps, steps, relres, st);
  cudaSetDevice(cur);
  return rc;
}

extern "C" int hmvm_b200_gcrm(hmvm_plan* plan, const void* b_dev, void* u_dev, int32_t max_steps, int32_t restart,
                              double eps, int32_t* steps, double* relres, void* stream) {
  hmvm_plan_info info;
  int rc = hmvm_b200_plan_get_info(plan, &info);
  if (rc) return rc;
  if (info.nd > 0 && (!b_dev || !u_dev)) return set_error(HMVM_EINVAL, "b or u is NULL");
  if (max_steps < 0 || !(eps >= 0.0)) return set_error(HMVM_EINVAL, "max_steps < 0 or eps not >= 0");
  if (restart < 1 || restart > kMaxRestart) return set_error(HMVM_EINVAL, "restart must be in 1..64");
  if (info.nd == 0) {
    if (steps) *steps = 0;
    if (relres) *relres = 0.0;
    return HMVM_OK;
  }
  int cur = 0;
  cudaGetDevice(&cur);
  if (cudaSetDevice(info.device) != cudaSuccess) return set_error(HMVM_ECUDA, "cannot select the plan's device");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (info.precision == HMVM_FP32)
    rc = gcrm_t<float>(plan, info.nd, static_cast<const float*>(b_dev), static_cast<float*>(u_dev), max_steps,
                       restart, eps, steps, relres, st);
  else
    rc = gcrm_t<double>(plan, info.nd, static_cast<const double*>(b_dev), static_cast<double*>(u_dev), max_steps,
                        restart, eps, steps, relres, st);
  cudaSetDevice(cur);
  return rc;
}
