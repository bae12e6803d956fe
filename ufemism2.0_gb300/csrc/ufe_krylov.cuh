// Krylov kernels: Jacobi-preconditioned BiCGStab in the form of PETSc's KSPBCGS with left
// preconditioning (the solver UFEMISM's solve_matrix_equation_CSR_PETSc hands its systems to,
// src/UPSY/basic/petsc_basic.f90:32-141, run with -ksp_type bcgs -pc_type jacobi).
//
// One iteration is three kernels:
//   k_p_spmv : p <- r - beta*omega*v + beta*p (also evaluated on the fly for gathered columns),
//              v <- D^-1 A p, partial (v, r^)                       -> alpha
//   k_s_spmv : s <- r - alpha*v (on the fly for gathered columns),
//              t <- D^-1 A s, partials (s,t), (t,t), (s,s)           -> omega
//   k_xr     : x <- x + alpha*p + omega*s,  r <- s - omega*t,
//              partials (r, r^), (r, r)                             -> convergence test, beta
// p and v are double-buffered by iteration parity, so the on-the-fly updates read old values.
// Every reduction is the deterministic last-block sum of ufe_work.cuh; kernels loop over their
// rows with a grid stride so the grid never exceeds the partial-sum capacity.
#pragma once

#include <math_constants.h>

#include <type_traits>

#include "ufe_dword.cuh"
#include "ufe_work.cuh"

template <class V> struct ScalarOf { using T = double; };
template <> struct ScalarOf<float2> { using T = float; };
template <> struct ScalarOf<double2> { using T = double; };
template <> struct ScalarOf<dw2> { using T = dw; };

// ---- vector element helpers ---------------------------------------------------------------
// The Krylov arithmetic uses explicit fused multiply-adds: FP64 instructions are the scarce
// resource on GB300, and these sums need no bitwise agreement with the reference.
__device__ __forceinline__ double v_dot(double2 a, double2 b) { return fma(a.y, b.y, a.x * b.x); }
__device__ __forceinline__ double v_dot(float2 a, float2 b) { return (double)fmaf(a.y, b.y, a.x * b.x); }
__device__ __forceinline__ double v_dot(double a, double b) { return a * b; }
__device__ __forceinline__ double2 v_mul(double2 d, double2 y) { return make_double2(d.x * y.x, d.y * y.y); }
__device__ __forceinline__ float2 v_mul(float2 d, float2 y) { return make_float2(d.x * y.x, d.y * y.y); }
__device__ __forceinline__ double v_mul(double d, double y) { return d * y; }
template <class V> __device__ __forceinline__ V v_zero();
template <> __device__ __forceinline__ double2 v_zero<double2>() { return make_double2(0.0, 0.0); }
template <> __device__ __forceinline__ float2 v_zero<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ double v_zero<double>() { return 0.0; }
template <> __device__ __forceinline__ dw2 v_zero<dw2>() { return dw2{make_float4(0.f, 0.f, 0.f, 0.f)}; }
// p_new = r - (beta*omega)*v + beta*p   (PETSc VecAXPBYPCZ(P, 1, -beta*omega, beta, R, V))
__device__ __forceinline__ double2 v_pupd(double2 r, double bw, double2 v, double beta, double2 p) {
  return make_double2(fma(beta, p.x, fma(-bw, v.x, r.x)), fma(beta, p.y, fma(-bw, v.y, r.y)));
}
__device__ __forceinline__ float2 v_pupd(float2 r, float bw, float2 v, float beta, float2 p) {
  return make_float2(fmaf(beta, p.x, fmaf(-bw, v.x, r.x)), fmaf(beta, p.y, fmaf(-bw, v.y, r.y)));
}
__device__ __forceinline__ double v_pupd(double r, double bw, double v, double beta, double p) {
  return fma(beta, p, fma(-bw, v, r));
}
// r - a*v
__device__ __forceinline__ double2 v_sub_scaled(double2 r, double a, double2 v) {
  return make_double2(fma(-a, v.x, r.x), fma(-a, v.y, r.y));
}
__device__ __forceinline__ float2 v_sub_scaled(float2 r, float a, float2 v) {
  return make_float2(fmaf(-a, v.x, r.x), fmaf(-a, v.y, r.y));
}
__device__ __forceinline__ double v_sub_scaled(double r, double a, double v) { return fma(-a, v, r); }
// x + a*p: v_xupd in two steps
__device__ __forceinline__ double2 v_axpy(double2 x, double a, double2 p) {
  return make_double2(fma(a, p.x, x.x), fma(a, p.y, x.y));
}
// x + a*p + w*s
__device__ __forceinline__ double2 v_xupd(double2 x, double a, double2 p, double w, double2 s) {
  return make_double2(fma(w, s.x, fma(a, p.x, x.x)), fma(w, s.y, fma(a, p.y, x.y)));
}
__device__ __forceinline__ float2 v_xupd(float2 x, float a, float2 p, float w, float2 s) {
  return make_float2(fmaf(w, s.x, fmaf(a, p.x, x.x)), fmaf(w, s.y, fmaf(a, p.y, x.y)));
}
__device__ __forceinline__ double v_xupd(double x, double a, double p, double w, double s) {
  return fma(w, s, fma(a, p, x));
}
__device__ __forceinline__ double2 v_shfl_xor(double2 a, int o) {
  return make_double2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
}
__device__ __forceinline__ float2 v_shfl_xor(float2 a, int o) {
  return make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
}
__device__ __forceinline__ double v_shfl_xor(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ double2 v_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 v_add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double v_add(double a, double b) { return a + b; }

// ---- matrix access policies ---------------------------------------------------------------
// 2x2-block rows (one triangle = its u and v rows); blocks stored in MatReal (FP64 or FP32),
// vectors and accumulation in VecReal; L lanes per block row.
// Sliced ELL (one lane per row): block rows in slices of 32 (one warp), the k-th entry of row
// i at slot soff[i/32] + 32 k + i%32, so that a warp's loads of blocks and columns are
// contiguous.  Short rows are padded with zero blocks whose column is the row itself.
template <typename MatReal, typename VecReal, int L>
struct BsrMat {
  using Vec = typename std::conditional<sizeof(VecReal) == 8, double2, float2>::type;
  using Blk = typename std::conditional<sizeof(MatReal) == 8, double4, float4>::type;
  static constexpr int kLanes = L;
  int32_t items;
  const int32_t *__restrict__ ptr;
  const int32_t *__restrict__ col;
  const Blk *__restrict__ blk;
  const int32_t *__restrict__ soff = nullptr;   // sliced-ELL copy (L == 1), or null
  const int32_t *__restrict__ scol = nullptr;
  const Blk *__restrict__ sblk = nullptr;
  template <class G>
  __device__ __forceinline__ Vec row_partial(int i, int lane, G get) const {
    Vec y = v_zero<Vec>();
    if (L == 1 && soff) {
      const int sl = i >> 5;
      const int s0 = __ldg(soff + sl), w = (__ldg(soff + sl + 1) - s0) >> 5;
      const int base = s0 + (i & 31);
      int k = 0;
      for (; k + 4 <= w; k += 4) {   // four slots' loads in flight at once
        int c[4];
        Blk a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int slot = base + ((k + u) << 5);
          c[u] = __ldg(scol + slot);
          a[u] = sblk[slot];
        }
        Vec x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = get(c[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          y.x = fma(a[u].y, x[u].y, fma(a[u].x, x[u].x, y.x));
          y.y = fma(a[u].w, x[u].y, fma(a[u].z, x[u].x, y.y));
        }
      }
      for (; k < w; ++k) {
        const int slot = base + (k << 5);
        const Blk a = sblk[slot];
        const Vec x = get(__ldg(scol + slot));
        y.x = fma(a.y, x.y, fma(a.x, x.x, y.x));
        y.y = fma(a.w, x.y, fma(a.z, x.x, y.y));
      }
      return y;
    }
    int k2 = __ldg(ptr + i + 1);
    for (int k = __ldg(ptr + i) + lane; k < k2; k += L) {
      Blk a = blk[k];
      Vec x = get(__ldg(col + k));
      y.x = fma(a.y, x.y, fma(a.x, x.x, y.x));
      y.y = fma(a.w, x.y, fma(a.z, x.x, y.y));
    }
    return y;
  }
};

// FP32 2x2-block rows in difference form: y_i = sum_j A_ij (x_j - x_i) + S_i x_i with the row
// sums S_i = sum_j A_ij taken in FP64 at assembly.  For the smooth vectors of an elliptic
// operator, x_j - x_i is exact in FP32 (nearby values) and the products keep full relative
// precision, where the plain form loses the digits that cancel between diagonal and neighbours.
template <int L>
struct BsrDiffMat {
  using Vec = float2;
  using Blk = float4;
  static constexpr int kLanes = L;
  int32_t items;
  const int32_t *__restrict__ ptr;
  const int32_t *__restrict__ col;
  const float4 *__restrict__ blk;
  const float4 *__restrict__ rowsum;
  const int32_t *__restrict__ soff = nullptr;   // sliced-ELL copy (L == 1), or null
  const int32_t *__restrict__ scol = nullptr;
  const float4 *__restrict__ sblk = nullptr;
  template <class G>
  __device__ __forceinline__ float2 row_partial(int i, int lane, G get) const {
    const float2 xi = get(i);
    float2 y = make_float2(0.f, 0.f);
    if (lane == 0) {
      const float4 s = rowsum[i];
      y.x = fmaf(s.y, xi.y, s.x * xi.x);
      y.y = fmaf(s.w, xi.y, s.z * xi.x);
    }
    if (L == 1 && soff) {
      const int sl = i >> 5;
      const int s0 = __ldg(soff + sl), w = (__ldg(soff + sl + 1) - s0) >> 5;
      const int base = s0 + (i & 31);
      int k = 0;
      for (; k + 4 <= w; k += 4) {   // four slots' loads in flight at once
        int c[4];
        float4 a[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int slot = base + ((k + u) << 5);
          c[u] = __ldg(scol + slot);
          a[u] = sblk[slot];
        }
        float2 xj[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) xj[u] = get(c[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const float dx = xj[u].x - xi.x, dy = xj[u].y - xi.y;
          y.x = fmaf(a[u].y, dy, fmaf(a[u].x, dx, y.x));
          y.y = fmaf(a[u].w, dy, fmaf(a[u].z, dx, y.y));
        }
      }
      for (; k < w; ++k) {
        const int slot = base + (k << 5);
        const float4 a = sblk[slot];
        const float2 xj = get(__ldg(scol + slot));
        const float dx = xj.x - xi.x, dy = xj.y - xi.y;
        y.x = fmaf(a.y, dy, fmaf(a.x, dx, y.x));
        y.y = fmaf(a.w, dy, fmaf(a.z, dx, y.y));
      }
      return y;
    }
    int k2 = __ldg(ptr + i + 1);
    for (int k = __ldg(ptr + i) + lane; k < k2; k += L) {
      const float4 a = blk[k];
      const float2 xj = get(__ldg(col + k));
      const float dx = xj.x - xi.x, dy = xj.y - xi.y;
      y.x = fmaf(a.y, dy, fmaf(a.x, dx, y.x));
      y.y = fmaf(a.w, dy, fmaf(a.z, dx, y.y));
    }
    return y;
  }
};

// scalar CSR rows (the general matrix-equation solve), one lane per row
struct CsrMat {
  using Vec = double;
  static constexpr int kLanes = 1;
  int32_t items;
  const int32_t *__restrict__ ptr;
  const int32_t *__restrict__ col;
  const double *__restrict__ val;
  template <class G>
  __device__ __forceinline__ double row_partial(int i, int lane, G get) const {
    double y = 0.0;
    int k2 = __ldg(ptr + i + 1);
    for (int k = __ldg(ptr + i); k < k2; ++k) y = fma(__ldg(val + k), get(__ldg(col + k)), y);
    return y;
  }
};

template <class Vec>
struct KV {
  Vec *X, *R, *RP, *S, *T, *B;
  const Vec *dinv;
  Vec *P[2], *V[2];
};

// reduction sites (one ticket each)
enum : int {
  kSiteInit = 0, kSiteP, kSiteS, kSiteXR, kSiteResid, kSitePicard, kSiteAux, kSiteInner, kSiteCount
};

struct CondArg {
  cudaGraphConditionalHandle handle;
  int use;
};

__device__ __forceinline__ void set_cond(CondArg c, int value) {
  if (c.use) cudaGraphSetConditional(c.handle, value ? 1u : 0u);
}

template <int L, class Vec>
__device__ __forceinline__ Vec lane_reduce(Vec y) {
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) y = v_add(y, v_shfl_xor(y, o));
  return y;
}

// Lanes of one group must be in one warp: blockDim.x is a multiple of 32 and L divides 32.
#define KRYLOV_ROWS(M, i, lane)                                                                \
  const int lane = threadIdx.x % M::kLanes;                                                    \
  const int64_t gstride_ = ((int64_t)gridDim.x * blockDim.x) / M::kLanes;                      \
  const int64_t nrows_pad_ = ((mat.items + gstride_ - 1) / gstride_) * gstride_;               \
  for (int64_t i##_64 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / M::kLanes;          \
       i##_64 < nrows_pad_; i##_64 += gstride_)

// r = D^-1 (b - A x), r^ = r, p = v = 0; tests the initial residual (KSPConvergedDefault at
// iteration 0) and primes rho = (r, r^).
// With gate = 1 the kernel only runs when the scalars ask for an FP64 fallback solve.  With
// keep_tol = 1 (a restart inside one linear solve) the stopping tolerance set at the solve's start
// is kept.
template <class M>
__global__ void k_krylov_init(M mat, KV<typename M::Vec> v, KrylovScalars *ks, double rtol,
                              double abstol, int max_it, int x_is_zero, double *partials,
                              unsigned int *tickets, CondArg cond, int gate = 0, int keep_tol = 0) {
  using Vec = typename M::Vec;
  if (gate && !ks->fallback) {
    if (blockIdx.x == 0 && threadIdx.x == 0) set_cond(cond, 0);
    return;
  }
  double acc[2] = {0.0, 0.0};
  KRYLOV_ROWS(M, i, lane) {
    const int i = (int)i_64;
    const bool live = i < mat.items;
    Vec ax = v_zero<Vec>();
    if (!x_is_zero) {
      Vec part = live ? mat.row_partial(i, lane, [&](int j) { return v.X[j]; }) : v_zero<Vec>();
      ax = lane_reduce<M::kLanes>(part);
    }
    if (live && lane == 0) {
      Vec b = v.B[i], d = v.dinv[i];
      Vec r = v_mul(d, v_sub_scaled(b, 1.0, ax));
      Vec db = v_mul(d, b);
      v.R[i] = r;
      v.RP[i] = r;
      v.P[0][i] = v_zero<Vec>();
      v.V[0][i] = v_zero<Vec>();
      if (x_is_zero) v.X[i] = v_zero<Vec>();
      acc[0] += v_dot(r, r);
      acc[1] += v_dot(db, db);
    }
  }
  double tot[2];
  if (grid_sum<2>(acc, partials, tickets + kSiteInit, tot)) {
    double dp = sqrt(tot[0]);
    double bnorm = sqrt(tot[1]);
    double rnorm0 = bnorm != 0.0 ? bnorm : dp;
    KrylovScalars s = *ks;
    s.dp = dp;
    if (!gate && !keep_tol) {
      s.rnorm0 = rnorm0;
      s.ttol = fmax(rtol * rnorm0, abstol);   // a fallback or a restart keeps the solve's tolerance
    }
    s.fallback = 0;
    s.it = 0;
    s.max_it = max_it;
    s.rho = tot[0];
    s.rhoold = 1.0;
    s.alpha = 1.0;
    s.omegaold = 1.0;
    s.omega = 1.0;
    s.beta = s.rho;  // (rho/rhoold)*(alpha/omegaold) with rhoold = alpha = omegaold = 1
    s.status = UFE_OK;
    s.tbreak = 0;
    s.active = 1;
    if (isnan(dp)) { s.status = UFE_ERR_NAN; s.active = 0; }
    else if (dp <= s.ttol) s.active = 0;
    else if (s.rho == 0.0) { s.status = UFE_ERR_DIVERGED; s.active = 0; }
    *ks = s;
    set_cond(cond, s.active);
  }
}

// pre = 1: p (and, in k_s_spmv, s) were formed row by row beforehand (k_p_update, k_s_update) and
// the SpMV gathers them; pre = 0 forms them on the fly for every gathered column.  Both give the
// same values -- the same expression on the same inputs -- but the on-the-fly form repeats the
// update's FP64 work once per stored entry, which bounds a scalar CSR solve by the FP64 pipe.
template <class M>
__global__ void k_p_spmv(M mat, KV<typename M::Vec> v, KrylovScalars *ks, double *partials,
                         unsigned int *tickets, int pre = 0) {
  using Vec = typename M::Vec;
  using R = typename ScalarOf<Vec>::T;
  const KrylovScalars s = *ks;
  if (!s.active) return;
  const int cur = s.it & 1, nxt = cur ^ 1;
  const R beta = (R)s.beta, bw = (R)(s.beta * s.omegaold);
  const Vec *__restrict__ Po = v.P[cur];
  const Vec *__restrict__ Vo = v.V[cur];
  const Vec *__restrict__ Rr = v.R;
  const Vec *__restrict__ Pn = v.P[nxt];
  double acc[1] = {0.0};
  KRYLOV_ROWS(M, i, lane) {
    const int i = (int)i_64;
    const bool live = i < mat.items;
    Vec part = !live ? v_zero<Vec>()
               : pre ? mat.row_partial(i, lane, [&](int j) { return Pn[j]; })
                     : mat.row_partial(i, lane, [&](int j) { return v_pupd(Rr[j], bw, Vo[j], beta, Po[j]); });
    Vec y = lane_reduce<M::kLanes>(part);
    if (live && lane == 0) {
      if (!pre) v.P[nxt][i] = v_pupd(Rr[i], bw, Vo[i], beta, Po[i]);
      Vec vn = v_mul(v.dinv[i], y);
      v.V[nxt][i] = vn;
      acc[0] += v_dot(vn, v.RP[i]);
    }
  }
  double tot[1];
  if (grid_sum<1>(acc, partials, tickets + kSiteP, tot)) {
    KrylovScalars t = *ks;
    double d1 = tot[0];
    if (d1 == 0.0 || isnan(d1)) { t.status = isnan(d1) ? UFE_ERR_NAN : UFE_ERR_DIVERGED; t.active = 0; }
    else t.alpha = t.rho / d1;
    *ks = t;
  }
}

template <class M>
__global__ void k_s_spmv(M mat, KV<typename M::Vec> v, KrylovScalars *ks, double *partials,
                         unsigned int *tickets, int pre = 0) {
  using Vec = typename M::Vec;
  using R = typename ScalarOf<Vec>::T;
  const KrylovScalars s = *ks;
  if (!s.active) return;
  const int nxt = (s.it & 1) ^ 1;
  const R alpha = (R)s.alpha;
  const Vec *__restrict__ Vn = v.V[nxt];
  const Vec *__restrict__ Rr = v.R;
  const Vec *__restrict__ Sg = v.S;
  double acc[3] = {0.0, 0.0, 0.0};
  KRYLOV_ROWS(M, i, lane) {
    const int i = (int)i_64;
    const bool live = i < mat.items;
    Vec part = !live ? v_zero<Vec>()
               : pre ? mat.row_partial(i, lane, [&](int j) { return Sg[j]; })
                     : mat.row_partial(i, lane, [&](int j) { return v_sub_scaled(Rr[j], alpha, Vn[j]); });
    Vec y = lane_reduce<M::kLanes>(part);
    if (live && lane == 0) {
      Vec si = pre ? Sg[i] : v_sub_scaled(Rr[i], alpha, Vn[i]);
      Vec ti = v_mul(v.dinv[i], y);
      if (!pre) v.S[i] = si;
      v.T[i] = ti;
      acc[0] += v_dot(si, ti);
      acc[1] += v_dot(ti, ti);
      acc[2] += v_dot(si, si);
    }
  }
  double tot[3];
  if (grid_sum<3>(acc, partials, tickets + kSiteS, tot)) {
    KrylovScalars t = *ks;
    if (tot[1] == 0.0) {
      // t = 0: if s = 0 too, x + alpha p solves the system (bcgs.c's breakdown branch)
      if (tot[2] != 0.0) { t.status = UFE_ERR_DIVERGED; t.active = 0; }
      else { t.omega = 0.0; t.tbreak = 1; }
    } else if (isnan(tot[1])) {
      t.status = UFE_ERR_NAN; t.active = 0;
    } else {
      t.omega = tot[0] / tot[1];
    }
    *ks = t;
  }
}

// Row-wise p <- r - beta omega v + beta p and s <- r - alpha v for the pre form above.
template <class Vec>
__global__ void k_p_update(int64_t n, KV<Vec> v, const KrylovScalars *ks) {
  using R = typename ScalarOf<Vec>::T;
  const KrylovScalars s = *ks;
  if (!s.active) return;
  const int cur = s.it & 1, nxt = cur ^ 1;
  const R beta = (R)s.beta, bw = (R)(s.beta * s.omegaold);
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    v.P[nxt][i] = v_pupd(v.R[i], bw, v.V[cur][i], beta, v.P[cur][i]);
}

template <class Vec>
__global__ void k_s_update(int64_t n, KV<Vec> v, const KrylovScalars *ks) {
  using R = typename ScalarOf<Vec>::T;
  const KrylovScalars s = *ks;
  if (!s.active) return;
  const int nxt = (s.it & 1) ^ 1;
  const R alpha = (R)s.alpha;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    v.S[i] = v_sub_scaled(v.R[i], alpha, v.V[nxt][i]);
}

template <class M>
__global__ void k_xr(M mat, KV<typename M::Vec> v, KrylovScalars *ks, double *partials,
                     unsigned int *tickets, CondArg cond) {
  using Vec = typename M::Vec;
  using R = typename ScalarOf<Vec>::T;
  const KrylovScalars s = *ks;
  if (!s.active) {
    // an earlier kernel of this iteration stopped the solve: end the loop here as well, so the
    // while-node never repeats an inactive body
    if (blockIdx.x == 0 && threadIdx.x == 0) set_cond(cond, 0);
    return;
  }
  const int nxt = (s.it & 1) ^ 1;
  const R alpha = (R)s.alpha, omega = (R)s.omega;
  double acc[2] = {0.0, 0.0};
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < mat.items; i += stride) {
    Vec pi = v.P[nxt][i], si = v.S[i], ti = v.T[i];
    v.X[i] = v_xupd(v.X[i], alpha, pi, omega, si);
    Vec ri = v_sub_scaled(si, omega, ti);
    v.R[i] = ri;
    acc[0] += v_dot(ri, v.RP[i]);
    acc[1] += v_dot(ri, ri);
  }
  double tot[2];
  if (grid_sum<2>(acc, partials, tickets + kSiteXR, tot)) {
    KrylovScalars t = *ks;
    t.it += 1;
    t.total_its += 1;
    double dp = sqrt(tot[1]);
    t.dp = dp;
    double rho_new = tot[0];
    t.rhoold = t.rho;
    t.omegaold = t.omega;
    t.rho = rho_new;
    if (t.tbreak) { t.active = 0; t.status = UFE_OK; t.dp = 0.0; }
    else if (isnan(dp)) { t.status = UFE_ERR_NAN; t.active = 0; }
    else if (dp <= t.ttol) { t.active = 0; }
    else if (dp >= 1e4 * t.rnorm0) { t.status = UFE_ERR_DIVERGED; t.active = 0; }
    else if (t.it >= t.max_it) { t.status = UFE_WARN_KRYLOV_MAXIT; t.active = 0; }
    else if (rho_new == 0.0) { t.status = UFE_ERR_DIVERGED; t.active = 0; }
    else t.beta = (t.rho / t.rhoold) * (t.alpha / t.omegaold);
    *ks = t;
    set_cond(cond, t.active);
  }
}

// Grid for the Krylov kernels: enough blocks to cover the rows once, capped so that the
// per-block partial sums fit the reduction area.
template <class M>
inline unsigned krylov_grid(const M &mat, int threads, int max_blocks) {
  int64_t lanes = (int64_t)mat.items * M::kLanes;
  int64_t b = (lanes + threads - 1) / threads;
  if (b > max_blocks) b = max_blocks;
  if (b < 1) b = 1;
  return (unsigned)b;
}

// ---- persistent BiCGStab: the whole iteration loop in one (co-resident) launch ----------------
// The same recurrence as k_p_spmv / k_s_spmv / k_xr, with the launches replaced by grid
// barriers.  After each phase every block writes its partial sums; after the barrier every block
// sums all blocks' partials in the same fixed order, so all blocks hold identical scalars and
// take identical decisions without another round trip.  The barrier's spin is bounded: a block
// that waits too long records the failure and every block leaves the loop.
constexpr int kPersistMaxBlocks = 8 * 152;
constexpr int kPersistSlots = 5;     // partial sums per block per phase

// The barrier counts arrivals monotonically within one launch: barrier k of a launch with G
// blocks is passed once the counter reaches k*G.  Each block's thread 0 adds its arrival with a
// release reduction (no round trip) and polls the counter with acquire loads, so the last
// arrival releases everyone after one L2 write and one read.  The counter must be zero when a
// persistent kernel starts: every launch site resets it (k_reset_gsync / k_inner_init) on the
// same stream just before.  `err` ends every later wait of the launch once one wait gave up.
struct __align__(128) GridSync {
  unsigned int count;
  unsigned int pad0[31];
  unsigned int gen;     // last stamp of the stamped exchanges (below); runs on across launches
  int err;
  unsigned int pad1[30];
};

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add_u32(unsigned int *p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// false (block-uniform) when the wait gave up.  `target` is thread 0's running arrival target
// (zero at kernel start).
__device__ __forceinline__ bool grid_barrier(GridSync *gs, unsigned int &target) {
  __shared__ int ok_s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    target += gridDim.x;
    __threadfence();
    red_release_add_u32(&gs->count, 1u);
    for (long long spins = 0; ld_acquire_u32(&gs->count) < target; ++spins) {
      if (spins > (1ll << 24) || *((volatile int *)&gs->err)) {
        ok = 0;
        atomicExch(&gs->err, 1);
        break;
      }
      if (spins > 4096) __nanosleep(64);
    }
    __threadfence();
    ok_s = ok;
  }
  __syncthreads();
  return ok_s != 0;
}

// block sum of NP values (fixed tree), written by thread 0 to part[blockIdx.x * NP + k]
template <int NP>
__device__ __forceinline__ void block_partials(double *acc, double *part) {
  __shared__ double red[NP][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    double v = acc[k];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[k][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      double v = lane < nw ? red[k][lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) part[(int64_t)blockIdx.x * NP + k] = v;
    }
  }
}

// every block: the sum over all blocks' partials in one fixed order (warp 0; broadcast)
template <int NP>
__device__ __forceinline__ void all_partials(const double *part, double *tot) {
  __shared__ double res[NP];
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
#pragma unroll
    for (int k = 0; k < NP; ++k) {
      double v = 0.0;
      for (int b = lane; b < (int)gridDim.x; b += 32) v += __ldcg(part + (int64_t)b * NP + k);
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) res[k] = v;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NP; ++k) tot[k] = res[k];
}

// Starts from the state k_krylov_init / k_inner_init left in *ks (and P[0], V[0]); runs until the
// scalars stop the solve; leaves x, r, the counters and the status as the three-kernel loop does.
constexpr int kPersistThreads = 1024;   // one block per SM

template <class M>
__global__ void __launch_bounds__(kPersistThreads) k_bicgstab_persist(M mat, KV<typename M::Vec> v, KrylovScalars *ks,
                                                          double *part, GridSync *gs) {
  using Vec = typename M::Vec;
  using R = typename ScalarOf<Vec>::T;
  KrylovScalars s = *ks;
  if (!s.active) return;
  double *partP = part, *partS = part + kPersistMaxBlocks * kPersistSlots,
         *partX = part + 2 * kPersistMaxBlocks * kPersistSlots;
  unsigned int gen = 0;   // barrier arrival target (thread 0)
  const int lane0 = threadIdx.x % M::kLanes;
  const int64_t gstride = ((int64_t)gridDim.x * blockDim.x) / M::kLanes;
  const int64_t nrows_pad = ((mat.items + gstride - 1) / gstride) * gstride;
  const int64_t row0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / M::kLanes;
  bool ok = true;
  while (s.active) {
    const int cur = s.it & 1, nxt = cur ^ 1;
    // -- p <- r - beta omega v + beta p;  v <- D^-1 A p;  (v, r^)
    {
      const R beta = (R)s.beta, bw = (R)(s.beta * s.omegaold);
      const Vec *__restrict__ Po = v.P[cur];
      const Vec *__restrict__ Vo = v.V[cur];
      const Vec *__restrict__ Rr = v.R;
      double acc[1] = {0.0};
      for (int64_t i64 = row0; i64 < nrows_pad; i64 += gstride) {
        const int i = (int)i64;
        const bool live = i < mat.items;
        Vec pt = live ? mat.row_partial(i, lane0, [&](int j) { return v_pupd(Rr[j], bw, Vo[j], beta, Po[j]); })
                      : v_zero<Vec>();
        Vec y = lane_reduce<M::kLanes>(pt);
        if (live && lane0 == 0) {
          v.P[nxt][i] = v_pupd(Rr[i], bw, Vo[i], beta, Po[i]);
          const Vec vn = v_mul(v.dinv[i], y);
          v.V[nxt][i] = vn;
          acc[0] += v_dot(vn, v.RP[i]);
        }
      }
      block_partials<1>(acc, partP);
      if (!(ok = grid_barrier(gs, gen))) break;
      double tot[1];
      all_partials<1>(partP, tot);
      const double d1 = tot[0];
      if (d1 == 0.0 || isnan(d1)) {
        s.status = isnan(d1) ? UFE_ERR_NAN : UFE_ERR_DIVERGED;
        s.active = 0;
        break;
      }
      s.alpha = s.rho / d1;
    }
    // -- s <- r - alpha v;  t <- D^-1 A s;  (s,t), (t,t), (s,s)
    {
      const R alpha = (R)s.alpha;
      const Vec *__restrict__ Vn = v.V[nxt];
      const Vec *__restrict__ Rr = v.R;
      double acc[3] = {0.0, 0.0, 0.0};
      for (int64_t i64 = row0; i64 < nrows_pad; i64 += gstride) {
        const int i = (int)i64;
        const bool live = i < mat.items;
        Vec pt = live ? mat.row_partial(i, lane0, [&](int j) { return v_sub_scaled(Rr[j], alpha, Vn[j]); })
                      : v_zero<Vec>();
        Vec y = lane_reduce<M::kLanes>(pt);
        if (live && lane0 == 0) {
          const Vec si = v_sub_scaled(Rr[i], alpha, Vn[i]);
          const Vec ti = v_mul(v.dinv[i], y);
          v.S[i] = si;
          v.T[i] = ti;
          acc[0] += v_dot(si, ti);
          acc[1] += v_dot(ti, ti);
          acc[2] += v_dot(si, si);
        }
      }
      block_partials<3>(acc, partS);
      if (!(ok = grid_barrier(gs, gen))) break;
      double tot[3];
      all_partials<3>(partS, tot);
      if (tot[1] == 0.0) {
        if (tot[2] != 0.0) { s.status = UFE_ERR_DIVERGED; s.active = 0; break; }
        s.omega = 0.0;
        s.tbreak = 1;
      } else if (isnan(tot[1])) {
        s.status = UFE_ERR_NAN;
        s.active = 0;
        break;
      } else {
        s.omega = tot[0] / tot[1];
      }
    }
    // -- x <- x + alpha p + omega s;  r <- s - omega t;  (r, r^), (r, r)
    {
      const R alpha = (R)s.alpha, omega = (R)s.omega;
      double acc[2] = {0.0, 0.0};
      const int64_t stride = (int64_t)gridDim.x * blockDim.x;
      for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < mat.items; i += stride) {
        const Vec pi = v.P[nxt][i], si = v.S[i], ti = v.T[i];
        v.X[i] = v_xupd(v.X[i], alpha, pi, omega, si);
        const Vec ri = v_sub_scaled(si, omega, ti);
        v.R[i] = ri;
        acc[0] += v_dot(ri, v.RP[i]);
        acc[1] += v_dot(ri, ri);
      }
      block_partials<2>(acc, partX);
      if (!(ok = grid_barrier(gs, gen))) break;
      double tot[2];
      all_partials<2>(partX, tot);
      s.it += 1;
      s.total_its += 1;
      const double dp = sqrt(tot[1]);
      s.dp = dp;
      const double rho_new = tot[0];
      s.rhoold = s.rho;
      s.omegaold = s.omega;
      s.rho = rho_new;
      if (s.tbreak) { s.active = 0; s.status = UFE_OK; s.dp = 0.0; }
      else if (isnan(dp)) { s.status = UFE_ERR_NAN; s.active = 0; }
      else if (dp <= s.ttol) { s.active = 0; }
      else if (dp >= 1e4 * s.rnorm0) { s.status = UFE_ERR_DIVERGED; s.active = 0; }
      else if (s.it >= s.max_it) { s.status = UFE_WARN_KRYLOV_MAXIT; s.active = 0; }
      else if (rho_new == 0.0) { s.status = UFE_ERR_DIVERGED; s.active = 0; }
      else s.beta = (s.rho / s.rhoold) * (s.alpha / s.omegaold);
    }
  }
  if (!ok) {
    s.status = UFE_ERR_DEVICE;
    s.active = 0;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *ks = s;
}

// ---- persistent BiCGStab with shared-memory neighbourhoods (FP32 inner and FP64 solves) --------
// Block b owns the contiguous block rows [b*rpb, (b+1)*rpb) (whole sliced-ELL slices; the rows are
// in Z order, so they form a compact patch of the mesh).  Each SpMV phase first stages, into
// shared memory, the vector its rows read: its own rows (coalesced) and the patch's halo rows
// (listed once per mesh), computing the on-the-fly update (p, or s = r - alpha v) once per staged
// entry; the rows then read neighbours from shared memory through per-slot local indices.
template <class Blk>
struct HaloMat {
  int32_t items;
  int32_t rpb;                          // rows per block (a multiple of 32)
  const int32_t *__restrict__ soff;     // sliced-ELL slice offsets
  const int32_t *__restrict__ lcol;     // local index (own rows, then halo) per slot
  const Blk *__restrict__ sblk;         // blocks per slot
  const float4 *__restrict__ rowsum;    // FP32 difference form: FP64 row sums rounded to FP32
  const int32_t *__restrict__ halo_off; // gridDim.x + 1
  const int32_t *__restrict__ halo_idx; // global rows of each block's halo
  const uint8_t *__restrict__ halo_pub; // rows that are in some block's halo
};
using HaloDiffMat = HaloMat<float4>;

// FP32 difference form: y_i = S_i x_i + sum_j A_ij (x_j - x_i)
__device__ __forceinline__ float2 halo_row(const HaloMat<float4> &m, int i, int il, const float2 *tab) {
  const float2 xi = tab[il];
  const float4 sr = m.rowsum[i];
  float2 y = make_float2(fmaf(sr.y, xi.y, sr.x * xi.x), fmaf(sr.w, xi.y, sr.z * xi.x));
  const int sl = i >> 5;
  const int s0 = __ldg(m.soff + sl), w = (__ldg(m.soff + sl + 1) - s0) >> 5;
  const int base = s0 + (i & 31);
  int k = 0;
  for (; k + 4 <= w; k += 4) {   // four slots' loads in flight at once
    int c[4];
    float4 a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int slot = base + ((k + u) << 5);
      c[u] = __ldg(m.lcol + slot);
      a[u] = __ldg(m.sblk + slot);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float2 xj = tab[c[u]];
      const float dx = xj.x - xi.x, dy = xj.y - xi.y;
      y.x = fmaf(a[u].y, dy, fmaf(a[u].x, dx, y.x));
      y.y = fmaf(a[u].w, dy, fmaf(a[u].z, dx, y.y));
    }
  }
  for (; k < w; ++k) {
    const int slot = base + (k << 5);
    const float4 a = __ldg(m.sblk + slot);
    const float2 xj = tab[__ldg(m.lcol + slot)];
    const float dx = xj.x - xi.x, dy = xj.y - xi.y;
    y.x = fmaf(a.y, dy, fmaf(a.x, dx, y.x));
    y.y = fmaf(a.w, dy, fmaf(a.z, dx, y.y));
  }
  return y;
}

// FP64 plain form, summed in the row's storage order
__device__ __forceinline__ double2 halo_row(const HaloMat<double4> &m, int i, int il, const double2 *tab) {
  double2 y = make_double2(0.0, 0.0);
  const int sl = i >> 5;
  const int s0 = __ldg(m.soff + sl), w = (__ldg(m.soff + sl + 1) - s0) >> 5;
  const int base = s0 + (i & 31);
  int k = 0;
  for (; k + 4 <= w; k += 4) {
    int c[4];
    double4 a[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int slot = base + ((k + u) << 5);
      c[u] = __ldg(m.lcol + slot);
      a[u] = m.sblk[slot];
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const double2 x = tab[c[u]];
      y.x = fma(a[u].y, x.y, fma(a[u].x, x.x, y.x));
      y.y = fma(a[u].w, x.y, fma(a[u].z, x.x, y.y));
    }
  }
  for (; k < w; ++k) {
    const int slot = base + (k << 5);
    const double4 a = m.sblk[slot];
    const double2 x = tab[__ldg(m.lcol + slot)];
    y.x = fma(a.y, x.y, fma(a.x, x.x, y.x));
    y.y = fma(a.w, x.y, fma(a.z, x.x, y.y));
  }
  return y;
}

// Double-word form (UFE_PREC_FP32_PAIR), summed in the row's storage order with Dot2
// accumulators: the FP64 plain form's arithmetic on the FP32 pipe.
__device__ __forceinline__ dw2 halo_row(const HaloMat<dwblk> &m, int i, int il, const dw2 *tab) {
  dw_acc yu, yv;
  const int sl = i >> 5;
  const int s0 = __ldg(m.soff + sl), w = (__ldg(m.soff + sl + 1) - s0) >> 5;
  const int base = s0 + (i & 31);
  int k = 0;
  for (; k + 2 <= w; k += 2) {   // two slots' loads in flight at once (register budget of 64)
    int c[2];
    dwblk a[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int slot = base + ((k + u) << 5);
      c[u] = __ldg(m.lcol + slot);
      a[u] = m.sblk[slot];
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float4 x = tab[c[u]].q;
      yu.mac(a[u].hi.x, a[u].lo.x, x.x, x.z);
      yu.mac(a[u].hi.y, a[u].lo.y, x.y, x.w);
      yv.mac(a[u].hi.z, a[u].lo.z, x.x, x.z);
      yv.mac(a[u].hi.w, a[u].lo.w, x.y, x.w);
    }
  }
  for (; k < w; ++k) {
    const int slot = base + (k << 5);
    const dwblk a = m.sblk[slot];
    const float4 x = tab[__ldg(m.lcol + slot)].q;
    yu.mac(a.hi.x, a.lo.x, x.x, x.z);
    yu.mac(a.hi.y, a.lo.y, x.y, x.w);
    yv.mac(a.hi.z, a.lo.z, x.x, x.z);
    yv.mac(a.hi.w, a.lo.w, x.y, x.w);
  }
  return make_dw2(yu.result(), yv.result());
}

// Per-thread dot-product accumulators of the persistent solve: FP64 for the FP64 and FP32 forms;
// Dot2 pairs for the double-word form, summed across the block in double-word arithmetic (FP32
// pipe) and rounded to FP64 once per block for the grid sums.
template <class Vec>
struct DotAcc {
  using Part = double;
  double v = 0.0;
  __device__ __forceinline__ void add(Vec a, Vec b) { v += v_dot(a, b); }
  __device__ __forceinline__ Part part() const { return v; }
};
template <>
struct DotAcc<dw2> {
  using Part = float2;   // (hi, lo)
  dw_acc a;
  __device__ __forceinline__ void add(dw2 x, dw2 y) {
    a.mac(x.q.x, x.q.z, y.q.x, y.q.z);
    a.mac(x.q.y, x.q.w, y.q.y, y.q.w);
  }
  __device__ __forceinline__ Part part() const {
    const dw t = a.result();
    return make_float2(t.hi, t.lo);
  }
  static __device__ __forceinline__ Part zero() { return make_float2(0.f, 0.f); }
};

// ---- grid-wide sums of the persistent kernels ---------------------------------------------------
// A phase ends with the sum of one or five values over all blocks.  Every block puts its partial sums into
// its own slots, stamped with the number of this exchange, and every block reads all blocks' slots until
// each carries the stamp: the partials' arrival is the barrier, so no counter is incremented and nothing
// is loaded after the wait (a counter barrier followed by loads took two more L2 round trips).  The slots
// exist kReplicas times, each read by its share of the blocks: 152 SMs polling one copy delay its
// writers (wait of the p-phase on 115k triangles, mean over blocks: 6,200 cycles with two copies, 4,600 with
// eight, 4,200 with sixteen).  All cross-block data is made of 64-bit words of 32 data bits and the 32-bit
// stamp, so a torn read is seen and needs no fence.  Stamps run on from GridSync::gen across launches;
// words are written again only after every block has passed the next exchange, that is, after all have
// read them.  Every wait is bounded: a thread that polls too long, or sees that another gave up, sets
// `err` and every block leaves its loop.
//
// GB300 issues an FP64 instruction of a warp in 64 cycles per quarter SM whatever its active mask
// (measured: 0.50 lanes/clk per quarter, 65-cycle latency, 565 per division, ~615 per square root), and an
// instruction line that is not in the SM's instruction cache costs hundreds.  So the sums keep FP64
// instructions few and spread over the quarters' warps, run one piece of code in all of them (separate
// code per warp made the s-phase's sums 5x slower), skip the tree levels that would only add zeros, and
// compare on bit patterns; loops off the critical path stay rolled.  Every sum keeps one fixed order:
// threads as a binary tree (t + 512, 256, ... 32, then xor 16 ... 1), blocks b, b + 32, ... per lane,
// then xor 16 ... 1.
struct __align__(16) ExSlot {   // one FP64 value
  unsigned long long lo, hi;
};
struct __align__(32) ExRow {    // one 16-byte vector entry
  unsigned long long w[4];
};
constexpr unsigned int kExchangePolls = 1u << 22;
constexpr int kHaloMaxBlocks = 160;
constexpr int kReplicas = 8;
constexpr size_t kExSlots = 2 * (size_t)kReplicas * kPersistSlots * kHaloMaxBlocks;   // p-phase, s-phase

__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_words(void *p, unsigned long long a, unsigned long long b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words(const void *p, unsigned long long &a, unsigned long long &b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ unsigned long long word(unsigned int data, unsigned int stamp) {
  return (unsigned long long)data | ((unsigned long long)stamp << 32);
}
__device__ __forceinline__ bool stamped(unsigned long long w, unsigned int stamp) { return (unsigned int)(w >> 32) == stamp; }

__device__ __forceinline__ void slot_publish(ExSlot *p, double x, unsigned int stamp) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  st_words(p, word((unsigned int)u, stamp), word((unsigned int)(u >> 32), stamp));
}
// true when the poll loop has to give up
__device__ __forceinline__ bool poll_expired(unsigned int &polls, GridSync *gs) {
  if (++polls >= kExchangePolls || ((polls & 255u) == 0u && *((volatile int *)&gs->err))) {
    atomicExch(&gs->err, 1);
    return true;
  }
  return false;
}
// the slots of one exchange: value k of block b in replica c
__device__ __forceinline__ int slot_index(int k, int b, int c) {
  return (c * kPersistSlots + k) * kHaloMaxBlocks + b;
}
// Waits for this exchange's words, two 16-byte items per thread at a time (one after the other, the second's
// round trip follows the first's): all blocks' np partials to sp[k * kHaloMaxBlocks + block] (shared memory),
// and (kHalo) the entries of the nhalo rows hg[] of `rows` to halo[].  False after a timeout.
template <bool kHalo>
__device__ __forceinline__ bool exchange_wait(int np, const ExSlot *slots, double *sp, const ExRow *rows,
                                              const int *hg, int nhalo, double *halo, unsigned int stamp,
                                              GridSync *gs) {
  const int ns = np * kHaloMaxBlocks, n = kHalo ? ns + 2 * nhalo : ns, G = (int)gridDim.x;
  slots += slot_index(0, 0, (int)blockIdx.x % kReplicas);
  bool ok = true;
  // item t: slot t = k * kHaloMaxBlocks + block, then halo row (t - ns) / 2's halves; null: nothing to wait for
  auto item = [&](int t) -> const void * {
    if (t < ns) return t % kHaloMaxBlocks < G ? (const void *)(slots + t) : nullptr;
    if (!kHalo) return nullptr;
    return t < n ? (const void *)(rows[hg[(t - ns) >> 1]].w + 2 * ((t - ns) & 1)) : nullptr;
  };
  auto put = [&](int t, unsigned long long a, unsigned long long b) {
    (!kHalo || t < ns ? sp : halo - ns)[t] = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
  };
#pragma unroll 1
  for (int t = threadIdx.x; t < n; t += 2 * (int)blockDim.x) {
    const int t2 = t + (int)blockDim.x;
    const void *p0 = item(t), *p1 = item(t2);
    unsigned long long a = 0, b = 0, c = 0, d = 0;
    unsigned int polls = 0;
    for (;;) {
      if (p0) ld_words(p0, a, b);
      if (p1) ld_words(p1, c, d);
      if ((!p0 || (stamped(a, stamp) && stamped(b, stamp))) && (!p1 || (stamped(c, stamp) && stamped(d, stamp)))) break;
      if (poll_expired(polls, gs)) {
        ok = false;
        break;
      }
    }
    put(t, a, b);
    if (t2 < n) put(t2, c, d);
  }
  return ok;
}
// the lane's part of the sum of value k over the blocks: blocks lane, lane + 32, ... in this order.  The trip
// count is the same in all lanes: shuffles after a loop that lanes leave one by one took ~450 cycles each.
__device__ __forceinline__ double lane_blocks(const double *sp, int k, int lane) {
  const double *q = sp + k * kHaloMaxBlocks;
  double v = q[lane];
#pragma unroll 1
  for (int b = 32; b < (int)gridDim.x; b += 32) v = lane + b < (int)gridDim.x ? v + q[lane + b] : v;
  return v;
}
// the warp's index in a register the compiler knows to be uniform: branches on it are, too
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
// A vector entry for the blocks that have its row in their halo.
template <class Vec>
__device__ __forceinline__ void row_publish(ExRow *p, Vec x, unsigned int stamp) {
  static_assert(sizeof(Vec) == 16, "16-byte vector entries");
  uint4 q;
  memcpy(&q, &x, 16);
  st_words(p->w, word(q.x, stamp), word(q.y, stamp));
  st_words(p->w + 2, word(q.z, stamp), word(q.w, stamp));
}
// FP64 butterfly sums of a (in lanes below 16) and b (in the others)
__device__ __forceinline__ double warp_fold_sum(double a, double b) {
  const bool up = threadIdx.x & 16;
  double v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double fp64_div(double a, double b) { return a / b; }
// Double-word sums.  Two butterflies' step in one addition: lanes with `bit` clear go on with a, the others
// with b (fold(a, a, bit) is a butterfly step).  A double-word addition is 20 instructions, so five sums are folded.
__device__ __forceinline__ dw dw_fold(dw a, dw b, int bit) {
  const bool up = threadIdx.x & bit;
  const dw keep(up ? b.hi : a.hi, up ? b.lo : a.lo), send(up ? a.hi : b.hi, up ? a.lo : b.lo);
  return dw_add(keep, dw(__shfl_xor_sync(0xffffffffu, send.hi, bit), __shfl_xor_sync(0xffffffffu, send.lo, bit)));
}
__device__ __forceinline__ dw dw_warp_sum(dw a) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = dw_fold(a, a, o);
  return a;
}

// Sum the first np (1 or 5) accumulators over the block's first nact threads (the others hold zero) and publish
// them.  scratch: np * min(nact, blockDim) doubles (FP64 parts) or np * 32 float2 (double-word parts).
// kFence: the block's other writes are read after the exchange and have to be visible before the sums are.
template <bool kFence, class Acc>
__device__ __forceinline__ void block_publish(int np, const Acc (&acc)[kPersistSlots], int nact, void *scratch,
                                              ExSlot *slots, unsigned int stamp) {
  using P = typename Acc::Part;
  const int tid = threadIdx.x, lane = tid & 31, warp = warp_index();
  if constexpr (std::is_same<P, double>::value) {
    double *t = static_cast<double *>(scratch);
    if (tid < nact) {
      t[tid] = acc[0].part();
      if (np == 5)
#pragma unroll
        for (int k = 1; k < 5; ++k) t[k * nact + tid] = acc[k].part();
    }
    __syncthreads();
#pragma unroll 1
    for (int st = 512; st >= 256; st >>= 1) {
      if (st >= nact) continue;
      if (tid < st && tid + st < nact)
#pragma unroll 1
        for (int k = 0; k < np; ++k) t[k * nact + tid] += t[k * nact + tid + st];
      __syncthreads();
    }
    // value k in warp k, so that each quarter of the SM has one; a fifth value folds into warp 0's butterfly
    if (warp < min(np, 4)) {
      const int n = min(nact, 256), nseg = (n + 31) >> 5;
      double v0 = 0.0, v = 0.0;
#pragma unroll 1
      for (int k = warp; k < np; k += 4) {
        v0 = v;
        const double *q = t + k * nact + lane;
        auto seg = [&](int j) { return lane + 32 * j < n ? q[32 * j] : 0.0; };
        double a = seg(0), b = nseg > 2 ? seg(2) : 0.0, c = nseg > 1 ? seg(1) : 0.0, d = nseg > 3 ? seg(3) : 0.0;
        if (nseg > 4) a += seg(4);
        if (nseg > 6) b += seg(6);
        if (nseg > 5) c += seg(5);
        if (nseg > 7) d += seg(7);
        if (nseg > 2) a += b;
        if (nseg > 3) c += d;
        v = nseg > 1 ? a + c : a;
      }
      const bool two = np == 5 && warp == 0;   // v0 is value 0 and v value 4
      v = warp_fold_sum(two ? v0 : v, v);
      // every lane holds the sum: lane c writes replica c (of value 4: lane 16 + c)
      if (kFence) fence_acq_rel_gpu();
      if (lane < kReplicas || (two && lane >= 16 && lane < 16 + kReplicas))
        slot_publish(slots + slot_index(warp + ((lane >> 4) << 2), blockIdx.x, lane & 15), v, stamp);
    }
  } else {
    float2 *red = static_cast<float2 *>(scratch);
    const int nw = (nact + 31) >> 5;
    if (warp < nw) {
      dw x[5];
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const float2 q = acc[k].part();
        x[k] = dw(q.x, q.y);
      }
      if (np == 1) {
        const dw v = dw_warp_sum(x[0]);
        if (lane == 0) red[warp] = make_float2(v.hi, v.lo);
      } else {
        // 8 double-word additions instead of 25: value 0 ends in lane 0, 1 in 16, 2 in 8, 3 in 24, 4 in 4
        const dw ab = dw_fold(x[0], x[1], 16), cd = dw_fold(x[2], x[3], 16), e = dw_fold(x[4], x[4], 16);
        const dw abcd = dw_fold(ab, cd, 8), e8 = dw_fold(e, e, 8);
        dw v = dw_fold(abcd, e8, 4);
        v = dw_fold(v, v, 2);
        v = dw_fold(v, v, 1);
        if ((lane & 7) == 0) red[((lane >> 4) + ((lane >> 3) & 1) * 2) * 32 + warp] = make_float2(v.hi, v.lo);
        if (lane == 4) red[4 * 32 + warp] = make_float2(v.hi, v.lo);
      }
    }
    __syncthreads();
    if (warp < np) {
      const float2 q = lane < nw ? red[warp * 32 + lane] : make_float2(0.f, 0.f);
      const dw v = dw_warp_sum(dw(q.x, q.y));
      if (kFence) fence_acq_rel_gpu();
      if (lane < kReplicas) slot_publish(slots + slot_index(warp, blockIdx.x, lane), v.to_double(), stamp);
    }
  }
}

// ---- the scalar recurrence, after an exchange -------------------------------------------------------
__device__ __forceinline__ bool bits_nan(double x) {
  return ((unsigned long long)__double_as_longlong(x) << 1) > 0xffe0000000000000ull;
}
__device__ __forceinline__ bool bits_zero(double x) { return ((unsigned long long)__double_as_longlong(x) << 1) == 0ull; }
// a <= b for values that are not negative and not NaN (their bit patterns order as they do)
__device__ __forceinline__ bool bits_le(double a, double b) {
  return (unsigned long long)__double_as_longlong(a) <= (unsigned long long)__double_as_longlong(b);
}

// coefficients in the solve's arithmetic: [0] beta, [1] beta * omega_old, [2] alpha, [3] omega
template <class R>
struct __align__(16) PhaseScalars {
  KrylovScalars s;
  int finish;         // 1 when the last iteration's x/r update is still to be applied
  double res2;        // |r|^2 of the last iteration, >= 0
  double lo2, hi2;    // lo2 < |r|^2 < hi2: |r| is certainly above ttol and below the divergence limit
  double tot[kPersistSlots];
  __align__(8) unsigned char rs_raw[4 * sizeof(R)];
  __device__ __forceinline__ R *rs() { return reinterpret_cast<R *>(rs_raw); }
  // thread 0, at the start
  __device__ __forceinline__ void open(const KrylovScalars *ks) {
    s = *ks;
    rs()[0] = (R)s.beta;
    rs()[1] = (R)(s.beta * s.omegaold);
    finish = 0;
    res2 = s.dp * s.dp;
    // squares that a relative margin of 1e-12 keeps clear of the roundings of the square and of the root;
    // where a square leaves the normal range every iteration takes the root (lo2 = inf or hi2 = 0)
    const double a = s.ttol * s.ttol * (1.0 + 1e-12), d = 1e4 * s.rnorm0, b = d * d * (1.0 - 1e-12);
    lo2 = (s.ttol == 0.0 || (a > 1e-290 && a < 1e300)) ? a : CUDART_INF;
    hi2 = (b > 1e-290 && b < 1e300) ? b : 0.0;
  }
};

// The stopping tests of an iteration whose squared residual norm does not decide them, or that ends the solve.
template <class R>
static __device__ __noinline__ void stop_tests(PhaseScalars<R> &ph, double res2, double rho_new, bool zero) {
  KrylovScalars &s = ph.s;
  const double dp = sqrt(res2);
  s.dp = dp;
  if (zero) { s.tbreak = 1; s.active = 0; s.status = UFE_OK; s.dp = 0.0; }
  else if (bits_nan(dp)) { s.status = UFE_ERR_NAN; s.active = 0; }
  else if (bits_le(dp, s.ttol)) { s.active = 0; }
  else if (bits_le(1e4 * s.rnorm0, dp)) { s.status = UFE_ERR_DIVERGED; s.active = 0; }
  else if (s.it >= s.max_it) { s.status = UFE_WARN_KRYLOV_MAXIT; s.active = 0; }
  else if (bits_zero(rho_new)) { s.status = UFE_ERR_DIVERGED; s.active = 0; }
}
template <class R>
static __device__ __noinline__ void stop_failed(PhaseScalars<R> &ph, int status) {
  ph.s.status = status;
  ph.s.active = 0;
  if (ph.s.it > 0) ph.s.dp = sqrt(ph.res2);
}

// The scalars after an exchange; every thread of the block calls it, and sees the result after it.
// P-phase: alpha from (v, r^).  S-phase: omega, rho, beta and the stopping tests from (s,t), (t,t), (s,s), (s,r^),
// (t,r^).  Four warps, one on each quarter of the SM, sum the values, the two of rho in one butterfly.  Warps 0
// and 1 form omega; warp 0 goes on to the next iteration's coefficients (both divisions of beta in one
// instruction, in two lanes) while warp 1 does the stopping tests, on the squared residual norm where that
// decides them: the root (~615 cycles) is taken only near a limit and in the iteration that stops.
template <class R>
__device__ __forceinline__ void after_exchange(PhaseScalars<R> &ph, const double *sp, bool s_phase) {
  const int warp = warp_index(), lane = threadIdx.x & 31;
  if (warp < (s_phase ? 4 : 1)) {   // one piece of code for all: instruction fetches are a cost here
    // warp 0 (s,t) or (v,r^), 1 (t,t), 2 (s,r^) and (t,r^), 3 (s,s)
    const int k = warp < 2 ? warp : 5 - warp;
    double a = 0.0, b = 0.0;
#pragma unroll 1
    for (int q = k;; q = 4) {
      a = b;
      b = lane_blocks(sp, q, lane);
      if (warp != 2 || q == 4) break;
    }
    const double v = warp_fold_sum(warp == 2 ? a : b, b);
    if (lane == 0) ph.tot[k] = v;
    if (warp == 2 && lane == 16) ph.tot[4] = v;
    if (warp >= 2) asm volatile("bar.arrive 2, 128;" ::: "memory");
  }
  if (warp < (s_phase ? 2 : 1)) {
    if (s_phase) asm volatile("bar.sync 1, 64;" ::: "memory");
    else __syncwarp();
    // P: alpha = rho / (v,r^);  S: omega = (s,t) / (t,t)
    const double st = ph.tot[0], den = ph.tot[s_phase ? 1 : 0];
    const bool zero = bits_zero(den), nan = bits_nan(den);
    const double w = (s_phase && zero) ? 0.0 : fp64_div(s_phase ? st : ph.s.rho, den);
    if (!s_phase) {
      const R a = (R)w;
      if (lane == 0) {
        ph.finish = 0;   // the staging applied the previous iteration's x/r update
        if (nan || zero) {
          stop_failed(ph, nan ? UFE_ERR_NAN : UFE_ERR_DIVERGED);
        } else {
          ph.s.alpha = w;
          ph.rs()[2] = a;
        }
      }
    } else {
      asm volatile("bar.sync 2, 128;" ::: "memory");
      const double ss = ph.tot[2], rho_new = ph.tot[3] - w * ph.tot[4];
      const bool fail = (zero && !bits_zero(ss)) || nan;
      if (warp == 0) {
        const double rho_old = ph.s.rho;
        const double q = fp64_div(lane == 0 ? rho_new : ph.s.alpha, lane == 0 ? rho_old : w);
        const double beta = __shfl_sync(0xffffffffu, q, 0) * __shfl_sync(0xffffffffu, q, 1);
        const double bw = beta * w;
        const R c = (R)(lane == 0 ? beta : lane == 1 ? bw : w);
        if (!fail) {
          if (lane < 3) ph.rs()[lane == 2 ? 3 : lane] = c;
          if (lane == 0) {
            ph.s.omega = w;
            ph.s.rhoold = rho_old;
            ph.s.omegaold = w;
            ph.s.rho = rho_new;
            ph.s.beta = beta;
          }
        }
      } else {
        // a negative difference of roundings is zero; an undefined one (an overflowed sum) stays undefined
        const double raw = ss - w * (2.0 * st - w * den), res2 = raw > 0.0 || bits_nan(raw) ? raw : 0.0;
        if (lane == 0) {
          if (fail) {
            stop_failed(ph, zero ? UFE_ERR_DIVERGED : UFE_ERR_NAN);
          } else {
            ph.finish = 1;   // this iteration's x/r update is due from here on
            ph.res2 = res2;
            const int it = ph.s.it + 1;
            ph.s.it = it;
            ph.s.total_its += 1;
            if (zero || it >= ph.s.max_it || bits_zero(rho_new) || bits_le(res2, ph.lo2) || bits_le(ph.hi2, res2))
              stop_tests(ph, res2, rho_new, zero);
          }
        }
      }
    }
  }
  __syncthreads();
}

// block 0, at the end: the result and the next launch's first stamp (every block read this launch's
// before its first exchange; after a timeout another block may be one exchange further)
__device__ __forceinline__ void persist_close(KrylovScalars &s, bool ok, KrylovScalars *ks, GridSync *gs,
                                              unsigned int stamp) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    if (!ok) {
      s.status = UFE_ERR_DEVICE;
      s.active = 0;
    }
    *ks = s;
    gs->gen = stamp + 4u;
  }
}

// The whole BiCGStab solve in one launch (one 1024-thread block per SM): each block owns the
// contiguous rows [blockIdx.x * rpb, ...) and stages its patch (own rows, then halo rows) in
// shared memory for the two SpMVs.  The scalar recurrence runs once per block, on the block's
// shared copy of the scalars; the other threads read the coefficients of the next phase from
// shared memory, already in the solve's arithmetic (FP64, FP32 or double-word).
//
// Two grid-wide reductions per iteration instead of three.  The s-phase also forms (s, r^) and
// (t, r^), so the scalars of r_{k+1} = s - omega t follow without reducing over r:
//   (r_{k+1}, r^) = (s, r^) - omega (t, r^),   |r_{k+1}|^2 = (s, s) - omega (2 (s, t) - omega (t, t)),
// and the x/r update of iteration k runs inside the p staging of iteration k+1 (r of a halo row
// is formed on the fly from its s and t; each row's owner writes x and r).  The iterates are
// those of PETSc's KSPBCGS; only the rounding of rho and of the residual norm differs.  The
// x/r update of the last iteration runs after the loop.
//
// This form takes any number of rows per block and keeps every vector in global memory; meshes of at
// most one row per thread run k_bicgstab_resident below.
template <class Vec, class Blk>
__global__ void __launch_bounds__(kPersistThreads) k_bicgstab_halo(HaloMat<Blk> m, KV<Vec> v, KrylovScalars *ks,
                                                                   ExSlot *slots, GridSync *gs) {
  using R = typename ScalarOf<Vec>::T;
  constexpr bool kDw = std::is_same<Vec, dw2>::value;
  extern __shared__ __align__(16) unsigned char tab_raw[];
  Vec *tab = reinterpret_cast<Vec *>(tab_raw);
  __shared__ PhaseScalars<R> ph;
  __shared__ double sp[kPersistSlots * kHaloMaxBlocks];
  __shared__ __align__(16) unsigned char scratch[kDw ? kPersistSlots * 32 * sizeof(float2)
                                                     : kPersistSlots * kPersistThreads * sizeof(double)];
  if (threadIdx.x == 0) ph.open(ks);
  __syncthreads();
  if (!ph.s.active) return;
  ExSlot *slotP = slots, *slotS = slots + kReplicas * kPersistSlots * kHaloMaxBlocks;
  unsigned int stamp = *((volatile unsigned int *)&gs->gen);
  const int r0 = blockIdx.x * m.rpb;
  const int r1 = min(m.items, r0 + m.rpb);
  const int own = max(r1 - r0, 0);
  const int nact = min(own, (int)blockDim.x);
  const int h0 = __ldg(m.halo_off + blockIdx.x);
  const int nloc = own + (__ldg(m.halo_off + blockIdx.x + 1) - h0);
  bool ok = true, pending = false;   // pending: iteration k-1's x/r update not yet applied
  for (;;) {
    const int cur = ph.s.it & 1, nxt = cur ^ 1;
    // -- [x <- x + alpha p + omega s; r <- s - omega t]  p <- r - beta omega v + beta p (staged);
    //    v <- D^-1 A p;  (v, r^)
    {
      const R beta = ph.rs()[0], bw = ph.rs()[1], ap = ph.rs()[2], wp = ph.rs()[3];
      const Vec *__restrict__ Po = v.P[cur];
      const Vec *__restrict__ Vo = v.V[cur];
      for (int e = threadIdx.x; e < nloc; e += blockDim.x) {
        const int g = e < own ? r0 + e : __ldg(m.halo_idx + h0 + e - own);
        const Vec po = Po[g];
        Vec r;
        if (pending) {
          const Vec sg = v.S[g];
          r = v_sub_scaled(sg, wp, v.T[g]);
          if (e < own) {
            v.X[g] = v_xupd(v.X[g], ap, po, wp, sg);
            v.R[g] = r;
          }
        } else {
          r = v.R[g];
        }
        const Vec pn = v_pupd(r, bw, Vo[g], beta, po);
        tab[e] = pn;
        if (e < own) v.P[nxt][g] = pn;
      }
      __syncthreads();
      DotAcc<Vec> acc[kPersistSlots];
      for (int il = threadIdx.x; il < own; il += blockDim.x) {
        const int i = r0 + il;
        const Vec vn = v_mul(v.dinv[i], halo_row(m, i, il, tab));
        v.V[nxt][i] = vn;
        acc[0].add(vn, v.RP[i]);
      }
      ++stamp;
      block_publish<true>(1, acc, nact, scratch, slotP, stamp);
      ok = exchange_wait<false>(1, slotP, sp, nullptr, nullptr, 0, nullptr, stamp, gs);
      fence_acq_rel_gpu();
      if (!(ok = __syncthreads_and(ok) != 0)) break;
      after_exchange(ph, sp, false);
      if (!ph.s.active) break;
    }
    // -- s <- r - alpha v (staged);  t <- D^-1 A s;  (s,t), (t,t), (s,s), (s,r^), (t,r^)
    {
      const R alpha = ph.rs()[2];
      const Vec *__restrict__ Vn = v.V[nxt];
      for (int e = threadIdx.x; e < nloc; e += blockDim.x) {
        const int g = e < own ? r0 + e : __ldg(m.halo_idx + h0 + e - own);
        const Vec sv = v_sub_scaled(v.R[g], alpha, Vn[g]);
        tab[e] = sv;
        if (e < own) v.S[g] = sv;
      }
      __syncthreads();
      DotAcc<Vec> acc[5];
      for (int il = threadIdx.x; il < own; il += blockDim.x) {
        const int i = r0 + il;
        const Vec si = tab[il];
        const Vec ti = v_mul(v.dinv[i], halo_row(m, i, il, tab));
        v.T[i] = ti;
        const Vec rp = v.RP[i];
        acc[0].add(si, ti);
        acc[1].add(ti, ti);
        acc[2].add(si, si);
        acc[3].add(si, rp);
        acc[4].add(ti, rp);
      }
      ++stamp;
      block_publish<true>(5, acc, nact, scratch, slotS, stamp);
      ok = exchange_wait<false>(5, slotS, sp, nullptr, nullptr, 0, nullptr, stamp, gs);
      fence_acq_rel_gpu();
      if (!(ok = __syncthreads_and(ok) != 0)) break;
      after_exchange(ph, sp, true);
      if (!ph.s.active) break;
      pending = true;
    }
  }
  // the x/r update of the last iteration
  if (ok && ph.finish) {
    const R alpha = ph.rs()[2], omega = ph.rs()[3];
    const int nxt = ((ph.s.it - 1) & 1) ^ 1;   // the parity p was written with in that iteration
    for (int il = threadIdx.x; il < own; il += blockDim.x) {
      const int i = r0 + il;
      const Vec si = v.S[i];
      v.X[i] = v_xupd(v.X[i], alpha, v.P[nxt][i], omega, si);
      v.R[i] = v_sub_scaled(si, omega, v.T[i]);
    }
  }
  persist_close(ph.s, ok, ks, gs, stamp);
}

// ---- one row per thread: the vectors and as much of the matrix as fits stay on the SM ---------------
// One matrix row's sum, block by block in storage order (the halves of a block as stored: 16 bytes each).
template <class Vec>
struct RowSum;
template <>
struct RowSum<double2> {
  double2 y = make_double2(0.0, 0.0);
  __device__ __forceinline__ void mac(uint4 h0, uint4 h1, double2 x) {
    const double ax = __hiloint2double(h0.y, h0.x), ay = __hiloint2double(h0.w, h0.z);
    const double az = __hiloint2double(h1.y, h1.x), aw = __hiloint2double(h1.w, h1.z);
    y.x = fma(ay, x.y, fma(ax, x.x, y.x));
    y.y = fma(aw, x.y, fma(az, x.x, y.y));
  }
  __device__ __forceinline__ double2 result() const { return y; }
};
template <>
struct RowSum<dw2> {
  dw_acc yu, yv;
  __device__ __forceinline__ void mac(uint4 h, uint4 l, dw2 xx) {
    const float4 x = xx.q;
    yu.mac(__uint_as_float(h.x), __uint_as_float(l.x), x.x, x.z);
    yu.mac(__uint_as_float(h.y), __uint_as_float(l.y), x.y, x.w);
    yv.mac(__uint_as_float(h.z), __uint_as_float(l.z), x.x, x.z);
    yv.mac(__uint_as_float(h.w), __uint_as_float(l.w), x.y, x.w);
  }
  __device__ __forceinline__ dw2 result() const { return make_dw2(yu.result(), yv.result()); }
};

// Shared-memory layout of k_bicgstab_resident for a block shape; `depth` blocks per row are kept.
struct ResidentLayout {
  int rows, local, halo, slots, depth;   // largest numbers of a block: rows, patch entries, halo entries, slots;
                                         // blocks kept per row
  size_t scratch_bytes;            // block_publish's scratch
  __host__ __device__ size_t tab() const { return 0; }
  __host__ __device__ size_t vec() const { return tab() + 16ull * local; }              // x, r^, D^-1 of own rows
  __host__ __device__ size_t hvec() const { return vec() + 3 * 16ull * rows; }          // r, p, v, t of halo rows
  __host__ __device__ size_t hidx() const { return hvec() + 4 * 16ull * halo; }
  __host__ __device__ size_t scratch() const { return hidx() + (4ull * halo + 15) / 16 * 16; }
  __host__ __device__ size_t lcol() const { return scratch() + (scratch_bytes + 15) / 16 * 16; }
  __host__ __device__ size_t blocks() const { return lcol() + (2ull * slots + 15) / 16 * 16; }
  __host__ __device__ size_t bytes() const { return blocks() + 32ull * depth * rows; }
};

// k_bicgstab_halo's iteration with one thread per own row: r, p, v and t of the row stay in the thread's
// registers, s in the staged table, x, r^, D^-1, the local column indices and the first `depth` blocks of
// every row in shared memory for the whole solve.  Only v and t of the rows in another block's halo leave
// the SM, as stamped entries that arrive during the exchange's wait: a halo row's r, p and s are formed again
// from them with the owner's operations on the owner's operands (same values) instead of being loaded.
// Same sums in the same order as k_bicgstab_halo.
//
// What bounds it: small meshes are a chain of latencies -- per iteration two L2 exchanges (~3,000 cycles with 152
// blocks, 1,400 with 37), the FP64 pipe (64 cycles per instruction and warp: 4 per stored block, so ~3,300 for a
// row of 13) and the scalar recurrence (~2,000 and ~3,300); the double-word form on 115k triangles is bound by
// the L2 stream of the blocks that do not fit.  Per iteration, with the counter-barrier kernel it replaces
// beside it: FP64 11.6 us (20.8) on 1,154 triangles, 14.0 (21.2) on 16,662, 35.0 (39.7) on 115,383; double-word
// 19.2 us (25.2) on 115,383.  Fewer threads leave more registers and loads in flight to each, so the launch
// takes 512, 768 or 1024 by the rows per block.
template <class Vec, class Blk, int NT>
__global__ void __launch_bounds__(NT, 1) k_bicgstab_resident(HaloMat<Blk> m, KV<Vec> v, KrylovScalars *ks,
                                                             ExSlot *slots, ExRow *xv, ExRow *xt, GridSync *gs,
                                                             ResidentLayout lay) {
  using R = typename ScalarOf<Vec>::T;
  static_assert(sizeof(Vec) == 16 && sizeof(Blk) == 32, "16-byte vector entries and 32-byte blocks");
  extern __shared__ __align__(16) unsigned char smem[];
  Vec *tab = reinterpret_cast<Vec *>(smem + lay.tab());
  Vec *sx = reinterpret_cast<Vec *>(smem + lay.vec());
  Vec *srp = sx + lay.rows, *sdinv = srp + lay.rows;
  Vec *hr = reinterpret_cast<Vec *>(smem + lay.hvec()), *hp = hr + lay.halo, *hv = hp + lay.halo, *ht = hv + lay.halo;
  int *hg = reinterpret_cast<int *>(smem + lay.hidx());
  void *scratch = smem + lay.scratch();
  uint16_t *slc = reinterpret_cast<uint16_t *>(smem + lay.lcol());
  uint4 *sb0 = reinterpret_cast<uint4 *>(smem + lay.blocks()), *sb1 = sb0 + (size_t)lay.depth * lay.rows;
  __shared__ PhaseScalars<R> ph;
  __shared__ double sp[kPersistSlots * kHaloMaxBlocks];
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid == 0) ph.open(ks);
  __syncthreads();
  if (!ph.s.active) return;
  ExSlot *slotP = slots, *slotS = slots + kReplicas * kPersistSlots * kHaloMaxBlocks;
  unsigned int stamp = *((volatile unsigned int *)&gs->gen);
  const int r0 = blockIdx.x * m.rpb;
  const int r1 = min(m.items, r0 + m.rpb);
  const int own = max(r1 - r0, 0);
  const int h0 = __ldg(m.halo_off + blockIdx.x);
  const int nloc = own + (__ldg(m.halo_off + blockIdx.x + 1) - h0);
  const bool mine = tid < own;
  const int nhalo = nloc - own, g = r0 + tid;
  const uint4 *__restrict__ gblk = reinterpret_cast<const uint4 *>(m.sblk);
  // this row's slots: global slot of its first block, their number, and the slice's place in slc
  int base = 0, width = 0, lbase = 0;
  if (mine) {
    const int sl = g >> 5;
    const int s0 = __ldg(m.soff + sl);
    base = s0 + lane;
    width = (__ldg(m.soff + sl + 1) - s0) >> 5;
    lbase = s0 - __ldg(m.soff + (r0 >> 5)) + lane;
  }
  const int kept = min(width, lay.depth);
  Vec r = v_zero<Vec>(), p = v_zero<Vec>(), vv = v_zero<Vec>(), tt = v_zero<Vec>(), x1 = v_zero<Vec>();
  {
    const int cur = ph.s.it & 1;
#pragma unroll 1
    for (int h = tid; h < nhalo; h += NT) {
      const int j = __ldg(m.halo_idx + h0 + h);
      hg[h] = j;
      hr[h] = v.R[j];
      hp[h] = v.P[cur][j];
      hv[h] = v.V[cur][j];
    }
    if (mine) {
      r = v.R[g];
      p = v.P[cur][g];
      vv = v.V[cur][g];
    }
    if (mine) {
      sx[tid] = v.X[g];
      srp[tid] = v.RP[g];
      sdinv[tid] = v.dinv[g];
#pragma unroll 1
      for (int k = 0; k < width; ++k) slc[lbase + 32 * k] = (uint16_t)__ldg(m.lcol + base + 32 * k);
#pragma unroll 1
      for (int k = 0; k < kept; ++k) {
        const int64_t q = 2ll * (base + 32 * k);
        sb0[k * lay.rows + tid] = gblk[q];
        sb1[k * lay.rows + tid] = gblk[q + 1];
      }
    }
  }
  __syncthreads();
  const bool pub = mine && __ldg(m.halo_pub + g);   // the row is in another block's halo
  auto spmv_row = [&]() {   // row `tid` times the staged vector
    RowSum<Vec> y;
    // the blocks that are not kept come last: the first of them is on its way during the kept ones
    uint4 a0, a1;
    const uint4 *gq = gblk + 2ll * (base + 32 * kept);
    if (kept < width) {
      a0 = __ldg(gq);
      a1 = __ldg(gq + 1);
    }
    const uint16_t *lc = slc + lbase;
    const uint4 *q0 = sb0 + tid, *q1 = sb1 + tid;
    constexpr int kUnroll = std::is_same<Vec, double2>::value ? 2 : 1;
#pragma unroll kUnroll
    for (int k = 0; k < kept; ++k, lc += 32, q0 += lay.rows, q1 += lay.rows) y.mac(*q0, *q1, tab[*lc]);
#pragma unroll 1
    for (int k = kept; k < width; ++k, lc += 32) {
      const uint4 c0 = a0, c1 = a1;
      gq += 64;
      if (k + 1 < width) {
        a0 = __ldg(gq);
        a1 = __ldg(gq + 1);
      }
      y.mac(c0, c1, tab[*lc]);
    }
    return y.result();
  };
  bool ok = true, s_phase = false;
  int pending = 0;   // iteration k-1's x/r update not yet applied
  // Two passes of one loop body per iteration, so that the product, the sums and the wait are fetched as one
  // piece of code each.
#pragma unroll 1
  for (;;) {
    if (!s_phase) {
      // [x <- x + alpha p + omega s; r <- s - omega t]  p <- r - beta omega v + beta p (staged)
      const R beta = ph.rs()[0], bw = ph.rs()[1], wp = ph.rs()[3];
#pragma unroll 1
      for (int h = NT - 1 - tid; h < nhalo; h += NT) {   // the last threads first: they have no own row
        Vec rh = hr[h];
        if (pending) {
          rh = v_sub_scaled(tab[own + h], wp, ht[h]);
          hr[h] = rh;
        }
        const Vec pn = v_pupd(rh, bw, hv[h], beta, hp[h]);
        hp[h] = pn;
        tab[own + h] = pn;
      }
      if (mine) {
        if (pending) {
          const Vec sg = tab[tid];
          r = v_sub_scaled(sg, wp, tt);
          sx[tid] = v_axpy(x1, wp, sg);
        }
        p = v_pupd(r, bw, vv, beta, p);
        tab[tid] = p;
      }
    } else {
      // s <- r - alpha v (staged)
      const R alpha = ph.rs()[2];
#pragma unroll 1
      for (int h = NT - 1 - tid; h < nhalo; h += NT) tab[own + h] = v_sub_scaled(hr[h], alpha, hv[h]);
      if (mine) tab[tid] = v_sub_scaled(r, alpha, vv);
    }
    __syncthreads();
    // v <- D^-1 A p;  (v, r^)      or      t <- D^-1 A s;  (s,t), (t,t), (s,s), (s,r^), (t,r^)
    ++stamp;
    DotAcc<Vec> acc[kPersistSlots];
    if (mine) {
      const Vec y = v_mul(sdinv[tid], spmv_row()), rp = srp[tid];
      if (pub) row_publish((s_phase ? xt : xv) + g, y, stamp);
      if (!s_phase) {
        vv = y;
        acc[0].add(y, rp);
      } else {
        tt = y;
        const Vec si = tab[tid];
        acc[0].add(si, y);
        acc[1].add(y, y);
        acc[2].add(si, si);
        acc[3].add(si, rp);
        acc[4].add(y, rp);
      }
    }
    const int np = s_phase ? 5 : 1;
    block_publish<false>(np, acc, own, scratch, s_phase ? slotS : slotP, stamp);
    if (mine && s_phase) x1 = v_axpy(sx[tid], ph.rs()[2], p);   // half of the x update, while the sums travel
    ok = exchange_wait<true>(np, s_phase ? slotS : slotP, sp, s_phase ? xt : xv, hg, nhalo,
                       reinterpret_cast<double *>(s_phase ? ht : hv), stamp, gs);
    if (!(ok = __syncthreads_and(ok) != 0)) break;
    after_exchange(ph, sp, s_phase);
    if (!ph.s.active) break;
    pending |= s_phase;
    s_phase = !s_phase;
    asm volatile("" : "+r"(pending));   // one copy of the body: the first passes are not peeled
  }
  if (mine) {
    Vec x = sx[tid];
    if (ok && ph.finish) {   // the x/r update of the last iteration
      const R omega = ph.rs()[3];
      const Vec si = tab[tid];
      x = v_axpy(x1, omega, si);
      r = v_sub_scaled(si, omega, tt);
    }
    v.X[g] = x;
    v.R[g] = r;
  }
  persist_close(ph.s, ok, ks, gs, stamp);
}

// ---- scalar CSR systems (solve_matrix_equation_CSR_PETSc, the ice-thickness step) --------------------------
// BiCGStab for a caller's matrix as one persistent launch.  There are no patches here, so p and s travel as
// stamped words (ExSlot) that the products' gathers wait for one by one: no barrier stands between forming a
// vector and multiplying by it, and no fence.  An iteration waits for its three sums only.
//
// The sums have the order of the kernels this replaces (k_p_spmv, k_s_spmv, k_xr with their last-block sums), so
// the iterates are the same to the bit: the rows belong to `nvirt` virtual blocks of 256 threads, row
// 256 b + t (+ 256 nvirt k) to thread t of virtual block b; 256 values are summed as warp butterflies, then a
// butterfly over the eight warps; the virtual blocks' sums are summed as values t, t + 256, ... of 256 threads
// in the same way.  A block of 256 q threads runs q virtual blocks at a time.
//
// What bounds it: latency (three exchanges of ~3,000 cycles, two gathers, the FP64 sums and scalars), and the
// vectors' and matrix's way from L2 for large systems.  60,000 rows of five entries: 19 us an iteration, 46 with five
// kernels (each ends in a last block's serial sums, 10 to 16 us however small the system) and a host check every
// eight; larger systems at kCsrPersistRows.
constexpr int kMaxVirt = 8 * 152;
constexpr int kCsrSums = 3;
constexpr size_t kCsrSet = (size_t)kReplicas * kCsrSums * kMaxVirt;   // slots of one exchange; two sets in turn

__device__ __forceinline__ ExSlot *csr_slot(ExSlot *set, int k, int b, int c) {
  return set + ((size_t)c * kCsrSums + k) * kMaxVirt + b;
}
// The sums of up to three values over the 256 threads of this thread's virtual block, as 8-lane groups of its first
// warp: lane 8 k + w of it returns value k's sum, for every w.  red: 32 doubles per virtual block of the block.
__device__ __forceinline__ double virt_sum(int np, double a, double b, double c, double *red) {
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 7, sub = threadIdx.x >> 8;
  double v;
  if (np == 1) {
    v = a + __shfl_xor_sync(0xffffffffu, a, 16);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
  } else {
    // two or three butterflies in one: after these steps lanes 0-7 carry a, 16-23 b and, of three, 8-15 and 24-31 c
    const bool up = lane & 16, mid = lane & 8;
    v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
    if (np == 3) {
      const double x = c + __shfl_xor_sync(0xffffffffu, c, 16);
      v = (mid ? x : v) + __shfl_xor_sync(0xffffffffu, mid ? v : x, 8);
    } else {
      v += __shfl_xor_sync(0xffffffffu, v, 8);
    }
  }
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  double *r = red + 32 * sub;
  if (lane == 0) r[w] = v;
  if (np > 1 && lane == 16) r[8 + w] = v;
  if (np == 3 && lane == 8) r[16 + w] = v;
  asm volatile("bar.sync %0, 256;" ::"r"(1 + sub) : "memory");   // the virtual block's warps
  double t = 0.0;
  if (w == 0) {
    t = r[lane];   // (lanes of values that are not asked for: unused)
    t += __shfl_xor_sync(0xffffffffu, t, 4);
    t += __shfl_xor_sync(0xffffffffu, t, 2);
    t += __shfl_xor_sync(0xffffffffu, t, 1);
  }
  return t;
}
// Waits for all virtual blocks' np sums and leaves the totals in tot[0 .. np); false (block-uniform) on a timeout.
__device__ __forceinline__ bool csr_exchange(int np, int nvirt, ExSlot *set, unsigned int stamp, GridSync *gs,
                                             double *sp, double *red, double *tot) {
  bool ok = true;
  const ExSlot *mine = csr_slot(set, 0, 0, (int)blockIdx.x % kReplicas);
  const int n = np * nvirt;
#pragma unroll 1
  for (int t = threadIdx.x; t < n; t += blockDim.x) {
    const int k = t / nvirt, b = t - k * nvirt;
    unsigned long long lo, hi;
    unsigned int polls = 0;
    for (;;) {
      ld_words(mine + k * kMaxVirt + b, lo, hi);
      if (stamped(lo, stamp) && stamped(hi, stamp)) break;
      if (poll_expired(polls, gs)) {
        ok = false;
        break;
      }
    }
    sp[k * kMaxVirt + b] = __longlong_as_double((long long)((lo & 0xffffffffull) | (hi << 32)));
  }
  if (!__syncthreads_and(ok)) return false;
  if (threadIdx.x < 256) {
    double v[kCsrSums] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int b = threadIdx.x; b < ((nvirt + 255) & ~255); b += 256)
#pragma unroll
      for (int k = 0; k < kCsrSums; ++k)
        if (k < np) v[k] = b < nvirt ? v[k] + sp[k * kMaxVirt + b] : v[k];
    const double t = virt_sum(np, v[0], v[1], v[2], red);
    if (threadIdx.x < 8 * np && (threadIdx.x & 7) == 0) tot[threadIdx.x >> 3] = t;
  }
  __syncthreads();
  return true;
}

// Row i times the vector of stamped words `in`, in storage order, four gathers in flight.
__device__ __forceinline__ double csr_row(const CsrMat &mat, int i, const ExSlot *in, unsigned int stamp, GridSync *gs,
                                          bool &ok) {
  double y = 0.0;
  const int k2 = __ldg(mat.ptr + i + 1);
#pragma unroll 1
  for (int k = __ldg(mat.ptr + i); k < k2; k += 4) {
    unsigned long long lo[4], hi[4];
    double a[4];
    int c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int q = min(k + j, k2 - 1);
      c[j] = __ldg(mat.col + q);
      a[j] = __ldg(mat.val + q);
    }
    unsigned int polls = 0;
    for (;;) {
      bool all = true;
#pragma unroll
      for (int j = 0; j < 4; ++j) ld_words(in + c[j], lo[j], hi[j]);
#pragma unroll
      for (int j = 0; j < 4; ++j) all = all && stamped(lo[j], stamp) && stamped(hi[j], stamp);
      if (all) break;
      if (poll_expired(polls, gs)) {
        ok = false;
        break;
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (k + j < k2) y = fma(a[j], __longlong_as_double((long long)((lo[j] & 0xffffffffull) | (hi[j] << 32))), y);
  }
  return y;
}

template <class M>
__global__ void __launch_bounds__(kPersistThreads) k_csr_persist(M mat, int nvirt, KV<typename M::Vec> v,
                                                                 KrylovScalars *ks, ExSlot *pw, ExSlot *sw,
                                                                 ExSlot *slots, GridSync *gs) {
  __shared__ PhaseScalars<double> ph;
  __shared__ double sp[kCsrSums * kMaxVirt];
  __shared__ double red[32 * kPersistThreads / 256];
  if (threadIdx.x == 0) ph.open(ks);
  __syncthreads();
  if (!ph.s.active) return;
  unsigned int stamp = *((volatile unsigned int *)&gs->gen);
  const int lane = threadIdx.x & 31, q = blockDim.x >> 8, sub = threadIdx.x >> 8;
  const int64_t gstride = (int64_t)nvirt * 256;
  double *P = v.P[0], *V = v.V[0];
  bool ok = true;
  int phase = 0;   // 0: p, v, alpha;  1: s, t, omega;  2: x, r, rho
  // every row of every virtual block of this block: body(row); once per virtual block afterwards: done(index)
  auto each_row = [&](auto &&body, auto &&done) {
#pragma unroll 1
    for (int b0 = blockIdx.x * q; b0 < nvirt; b0 += gridDim.x * q) {
      const int b = b0 + sub;
      if (b < nvirt)
#pragma unroll 1
        for (int64_t i = (int64_t)b * 256 + (threadIdx.x & 255); i < mat.items; i += gstride) body((int)i);
      done(b);
    }
  };
#pragma unroll 1
  for (;;) {
    ++stamp;
    ExSlot *set = slots + (stamp & 1u) * kCsrSet;
    const double beta = ph.rs()[0], bw = ph.rs()[1], alpha = ph.rs()[2], omega = ph.rs()[3];
    const int np = phase == 0 ? 1 : phase == 1 ? 3 : 2;
    if (phase < 2)
      each_row(
          [&](int i) {
            double x;
            if (phase == 0) {
              x = v_pupd(v.R[i], bw, V[i], beta, P[i]);
              P[i] = x;
            } else {
              x = v_sub_scaled(v.R[i], alpha, V[i]);
              v.S[i] = x;
            }
            slot_publish((phase == 0 ? pw : sw) + i, x, stamp);
          },
          [](int) {});
    double a0 = 0.0, a1 = 0.0, a2 = 0.0;
    each_row(
        [&](int i) {
          if (phase == 0) {
            const double vn = v_mul(v.dinv[i], csr_row(mat, i, pw, stamp, gs, ok));
            V[i] = vn;
            a0 += v_dot(vn, v.RP[i]);
          } else if (phase == 1) {
            const double si = v.S[i], ti = v_mul(v.dinv[i], csr_row(mat, i, sw, stamp, gs, ok));
            v.T[i] = ti;
            a0 += v_dot(si, ti);
            a1 += v_dot(ti, ti);
            a2 += v_dot(si, si);
          } else {
            const double si = v.S[i], ri = v_sub_scaled(si, omega, v.T[i]);
            v.X[i] = v_xupd(v.X[i], alpha, P[i], omega, si);
            v.R[i] = ri;
            a0 += v_dot(ri, v.RP[i]);
            a1 += v_dot(ri, ri);
          }
        },
        [&](int b) {
          const double t = virt_sum(np, a0, a1, a2, red);
          if (((threadIdx.x >> 5) & 7) == 0 && lane < 8 * np && b < nvirt)
            slot_publish(csr_slot(set, lane >> 3, b, lane & 7), t, stamp);
          a0 = a1 = a2 = 0.0;
          __syncthreads();   // red is used again
        });
    if (!(ok = __syncthreads_and(ok) != 0)) break;
    if (!(ok = csr_exchange(np, nvirt, set, stamp, gs, sp, red, ph.tot))) break;
    if (warp_index() == 0) {
      KrylovScalars &s = ph.s;
      const double t0 = ph.tot[0], t1 = ph.tot[1], t2 = ph.tot[2];
      if (phase == 0) {
        const bool nan = bits_nan(t0), stop = nan || bits_zero(t0);
        const double al = fp64_div(s.rho, t0);
        if (lane == 0) {
          if (stop) {
            s.status = nan ? UFE_ERR_NAN : UFE_ERR_DIVERGED;
            s.active = 0;
          } else {
            s.alpha = al;
            ph.rs()[2] = al;
          }
        }
      } else if (phase == 1) {
        const bool zero = bits_zero(t1), nan = bits_nan(t1), fail = (zero && !bits_zero(t2)) || nan;
        const double om = zero ? 0.0 : fp64_div(t0, t1);
        if (lane == 0) {
          if (fail) {
            s.status = zero ? UFE_ERR_DIVERGED : UFE_ERR_NAN;
            s.active = 0;
          } else {
            s.omega = om;
            s.tbreak = zero;
            ph.rs()[3] = om;
          }
        }
      } else {
        const double quo = fp64_div(lane == 0 ? t0 : s.alpha, lane == 0 ? s.rho : omega);
        const double be = __shfl_sync(0xffffffffu, quo, 0) * __shfl_sync(0xffffffffu, quo, 1);
        if (lane == 0) {
          s.it += 1;
          s.total_its += 1;
          s.rhoold = s.rho;
          s.omegaold = omega;
          s.rho = t0;
          ph.res2 = t1;
          if (s.tbreak || s.it >= s.max_it || bits_zero(t0) || bits_le(t1, ph.lo2) || bits_le(ph.hi2, t1))
            stop_tests(ph, t1, t0, s.tbreak != 0);
          s.beta = be;
          ph.rs()[0] = be;
          ph.rs()[1] = be * omega;
        }
      }
    }
    __syncthreads();
    if (!ph.s.active) break;
    phase = phase == 2 ? 0 : phase + 1;
  }
  if (threadIdx.x == 0 && ok && phase < 2 && ph.s.it > 0) ph.s.dp = sqrt(ph.res2);   // stopped between two norms
  persist_close(ph.s, ok, ks, gs, stamp);
}
