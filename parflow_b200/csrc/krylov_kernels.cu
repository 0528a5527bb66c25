// Grid vectors, deterministic reductions and the scalar side of GMRES.
//
// Reductions: a fixed grid of blocks writes one partial per block; the last
// block to finish (ticket counter) sums the partials in index order, so every
// result is bitwise reproducible run to run.  Results stay in device memory.
// The scalar GMRES steps (modified Gram-Schmidt bookkeeping, Givens QR,
// back substitution) run in one thread on device-resident scalars and follow
// pfsimulator/kinsol/iterativ.c:30-286 and spgmr.c:168-450.
#include "gpu_wait.cuh"
#include "pdl.cuh"
#include "pfgpu_kernels.h"
#include "nk_control.h"

namespace pfgpu {

// Four blocks per SM and four elements in flight per thread keep enough bytes
// in flight to stream at HBM bandwidth (projection with the next dot product at
// 512x512x50: 58 us against 76 with one element); short vectors take
// no more blocks than give each thread its four elements, since every block
// adds an atomic to the serial end of the reduction.
static const int RED_THREADS = 256;
static const int RED_BLOCKS = 592;  // 4 x 148 SMs
static const int RED_UNROLL = 4;
static int red_grid(long long n, int most) {
  const long long per = (long long)RED_THREADS * RED_UNROLL, need = (n + per - 1) / per;
  return (int)(need < 1 ? 1 : need < most ? need : most);
}

int reduce_blocks() { return RED_BLOCKS; }


struct OpDot {
  const double *a, *b;
  __device__ double operator()(long long i) const { return a[i] * b[i]; }
  __device__ static double comb(double x, double y) { return x + y; }
  __device__ static double init() { return 0.0; }
};
struct OpStep {  // |s| / (1/1 + |u|)  (KINScSteplength, kinsol.c:1490-1505)
  const double *s, *u;
  __device__ double operator()(long long i) const { return fabs(s[i] / (1.0 / 1.0 + fabs(u[i]))); }
  __device__ static double comb(double x, double y) { return x > y ? x : y; }
  __device__ static double init() { return 0.0; }
};

template <typename Op>
__global__ void __launch_bounds__(RED_THREADS) k_reduce(Op op, long long n, double *partial,
                                                        double *dst, unsigned int *ticket,
                                                        const int *gate) {
  pdl_enter();
  if (gate && !*gate) return;  // not needed this time
  __shared__ double sh[RED_THREADS / 32];
  __shared__ bool last;
  double acc = Op::init();
  const long long stride = (long long)gridDim.x * RED_THREADS;
  long long i = blockIdx.x * (long long)RED_THREADS + threadIdx.x;
  for (; i + (RED_UNROLL - 1) * stride < n; i += RED_UNROLL * stride) {
    double v[RED_UNROLL];
#pragma unroll
    for (int u = 0; u < RED_UNROLL; u++) v[u] = op(i + u * stride);
#pragma unroll
    for (int u = 0; u < RED_UNROLL; u++) acc = Op::comb(acc, v[u]);
  }
  for (; i < n; i += stride) acc = Op::comb(acc, op(i));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc = Op::comb(acc, __shfl_down_sync(0xffffffffu, acc, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = sh[0];
    for (int w = 1; w < RED_THREADS / 32; w++) b = Op::comb(b, sh[w]);
    if (gridDim.x == 1) {
      *dst = b;
      last = false;
    } else {
      partial[blockIdx.x] = b;
      __threadfence();
      unsigned int t = atomicAdd(ticket, 1u);
      last = (t == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (!last) return;
  // last block: ordered final sum
  __threadfence();
  double v = Op::init();
  for (int i = threadIdx.x; i < (int)gridDim.x; i += RED_THREADS) {
    double pv = ((volatile double *)partial)[i];
    v = (i == (int)threadIdx.x) ? pv : Op::comb(v, pv);
  }
  // fixed-order tree over threads
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = Op::comb(v, __shfl_down_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double r = sh[0];
    for (int w = 1; w < RED_THREADS / 32; w++) r = Op::comb(r, sh[w]);
    *dst = r;
    *ticket = 0u;
  }
}

template <typename Op>
static void reduce(Op op, long long n, double *dst, ReduceBuf rb, cudaStream_t st,
                   const int *gate = nullptr) {
  launch_pdl(k_reduce<Op>, dim3(red_grid(n, rb.blocks)), dim3(RED_THREADS), st, op, n, rb.partial, dst, rb.ticket, gate);
}

void launch_dot(const double *a, const double *b, long long n, double *dst, ReduceBuf rb,
                cudaStream_t st) {
  OpDot op{a, b};
  reduce(op, n, dst, rb, st);
}
void launch_steplen(const double *s, const double *u, long long n, double *dst, ReduceBuf rb,
                    cudaStream_t st, const int *gate) {
  OpStep op{s, u};
  reduce(op, n, dst, rb, st, gate);
}

// ---- fused multi-value reductions ------------------------------------------
// One pass over the vectors for several sums / maxima that the solver needs
// together; each value is reduced exactly like k_reduce (per-thread grid-
// stride accumulation, fixed-order block and final combination).  An op
// may also update a vector element-wise in the same pass (MGS axpy).
static const int RED_MAX_K = 4;

template <typename Op>
__global__ void __launch_bounds__(RED_THREADS) k_reduce_multi(Op op, long long n,
                                                              double *partial,
                                                              unsigned int *ticket) {
  constexpr int K = Op::K;
  pdl_enter();
  __shared__ double sh[K][RED_THREADS / 32];
  __shared__ bool last;
  Op o = op;
  o.setup();
  double acc[K];
#pragma unroll
  for (int q = 0; q < K; q++) acc[q] = 0.0;
  const long long stride = (long long)gridDim.x * RED_THREADS;
  long long i = blockIdx.x * (long long)RED_THREADS + threadIdx.x;
  for (; i + (RED_UNROLL - 1) * stride < n; i += RED_UNROLL * stride) {
    typename Op::In in[RED_UNROLL];
#pragma unroll
    for (int u = 0; u < RED_UNROLL; u++) in[u] = o.load(i + u * stride);
#pragma unroll
    for (int u = 0; u < RED_UNROLL; u++) o.acc(i + u * stride, in[u], acc);
  }
  for (; i < n; i += stride) o.acc(i, o.load(i), acc);
#pragma unroll
  for (int q = 0; q < K; q++) {
    double a = acc[q];
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) a = Op::comb(q, a, __shfl_down_sync(0xffffffffu, a, w));
    if ((threadIdx.x & 31) == 0) sh[q][threadIdx.x >> 5] = a;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < K; q++) {
      double b = sh[q][0];
      for (int w = 1; w < RED_THREADS / 32; w++) b = Op::comb(q, b, sh[q][w]);
      if (gridDim.x == 1)
        *o.dst[q] = b;
      else
        partial[q * gridDim.x + blockIdx.x] = b;
    }
    last = false;
    if (gridDim.x > 1) {
      __threadfence();
      unsigned int t = atomicAdd(ticket, 1u);
      last = (t == gridDim.x - 1);
    }
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int q = 0; q < K; q++) {
    double v = 0.0;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += RED_THREADS) {
      double pv = ((volatile double *)partial)[q * gridDim.x + i];
      v = (i == (int)threadIdx.x) ? pv : Op::comb(q, v, pv);
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) v = Op::comb(q, v, __shfl_down_sync(0xffffffffu, v, w));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[q][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < K; q++) {
      double r = sh[q][0];
      for (int w = 1; w < RED_THREADS / 32; w++) r = Op::comb(q, r, sh[q][w]);
      *o.dst[q] = r;
    }
    *ticket = 0u;
  }
}

__device__ __forceinline__ double comb_sum(double x, double y) { return x + y; }
__device__ __forceinline__ double comb_max(double x, double y) { return x > y ? x : y; }

// <vk, vk> and <v0, vk> (the first two dot products of ModifiedGS)
struct OpMgsFirst {
  static constexpr int K = 2;
  const double *vk, *v0;
  double *dst[K];
  struct In {
    double a, v;
  };
  __device__ void setup() {}
  __device__ In load(long long i) const { return In{vk[i], v0[i]}; }
  __device__ void acc(long long, const In &q, double *v) const {
    v[0] = v[0] + q.a * q.a;
    v[1] = v[1] + q.v * q.a;
  }
  __device__ static double comb(int, double x, double y) { return comb_sum(x, y); }
};
// y = y + sign * (*s) x, then <z, y> with the updated y (z = y when null):
// one ModifiedGS projection fused with the next dot product
struct OpAxpyDot {
  static constexpr int K = 1;
  double *y;
  const double *x, *s, *z;
  double sign, a;
  double *dst[K];
  struct In {
    double y, x, z;
  };
  __device__ void setup() { a = sign * (*s); }
  __device__ In load(long long i) const { return In{y[i], x[i], z ? z[i] : 0.0}; }
  __device__ void acc(long long i, const In &q, double *v) {
    const double yn = q.y + a * q.x;
    y[i] = yn;
    const double zi = z ? q.z : yn;
    v[0] = v[0] + zi * yn;
  }
  __device__ static double comb(int, double x, double y) { return comb_sum(x, y); }
};
// line-search inputs after the Newton direction p: <Jp, Jp>, <f, Jp>, <p, p>
// and max |p| / (1 + |u|)
struct OpLineSearchIn {
  static constexpr int K = 4;
  const double *jp, *f, *p, *u;
  double *dst[K];
  struct In {
    double j, p, f, u;
  };
  __device__ void setup() {}
  __device__ In load(long long i) const { return In{jp[i], p[i], f[i], u[i]}; }
  __device__ void acc(long long, const In &q, double *v) const {
    v[0] = v[0] + q.j * q.j;
    v[1] = v[1] + q.f * q.j;
    v[2] = v[2] + q.p * q.p;
    v[3] = comb_max(v[3], fabs(q.p / (1.0 / 1.0 + fabs(q.u))));
  }
  __device__ static double comb(int q, double x, double y) {
    return q == 3 ? comb_max(x, y) : comb_sum(x, y);
  }
};
// after a trial step: <f, f>, max |f| and max |unew - u| / (1 + |unew|)
struct OpStepNorms {
  static constexpr int K = 2;
  const double *f;
  double *dst[K];
  struct In {
    double f;
  };
  __device__ void setup() {}
  __device__ In load(long long i) const { return In{f[i]}; }
  __device__ void acc(long long, const In &q, double *v) const {
    v[0] = v[0] + q.f * q.f;
    v[1] = comb_max(v[1], fabs(q.f));
  }
  __device__ static double comb(int q, double x, double y) {
    return q == 0 ? comb_sum(x, y) : comb_max(x, y);
  }
};
// at KINSol's start: <u, u>, max |f|, <f, f>
struct OpInitNorms {
  static constexpr int K = 3;
  const double *u, *f;
  double *dst[K];
  struct In {
    double u, f;
  };
  __device__ void setup() {}
  __device__ In load(long long i) const { return In{u[i], f[i]}; }
  __device__ void acc(long long, const In &q, double *v) const {
    v[0] = v[0] + q.u * q.u;
    v[1] = comb_max(v[1], fabs(q.f));
    v[2] = v[2] + q.f * q.f;
  }
  __device__ static double comb(int q, double x, double y) {
    return q == 1 ? comb_max(x, y) : comb_sum(x, y);
  }
};

// <u, v>, <v, v> and sum |v| of a difference-quotient product (KINSpgmrAtimesDQ)
struct OpDQ {
  static constexpr int K = 3;
  const double *u, *v;
  double *dst[K];
  struct In {
    double u, v;
  };
  __device__ void setup() {}
  __device__ In load(long long i) const { return In{u[i], v[i]}; }
  __device__ void acc(long long, const In &q, double *s) const {
    s[0] = s[0] + q.u * q.v;
    s[1] = s[1] + q.v * q.v;
    s[2] = s[2] + fabs(q.v);
  }
  __device__ static double comb(int, double x, double y) { return comb_sum(x, y); }
};

template <typename Op>
static void reduce_multi(Op op, long long n, ReduceBuf rb, cudaStream_t st) {
  launch_pdl(k_reduce_multi<Op>, dim3(red_grid(n, rb.blocks)), dim3(RED_THREADS), st, op, n, rb.partial,
             rb.ticket);
}

int reduce_partials() { return RED_BLOCKS * RED_MAX_K; }

void launch_mgs_first(const double *vk, const double *v0, long long n, double *d_vk2,
                      double *d_h0, ReduceBuf rb, cudaStream_t st) {
  OpMgsFirst op{vk, v0, {d_vk2, d_h0}};
  reduce_multi(op, n, rb, st);
}
void launch_axpy_dot(double *y, const double *x, const double *s, double sign, const double *z,
                     long long n, double *dst, ReduceBuf rb, cudaStream_t st) {
  OpAxpyDot op{y, x, s, z, sign, 0.0, {dst}};
  reduce_multi(op, n, rb, st);
}
void launch_linesearch_inputs(const double *jp, const double *f, const double *p,
                              const double *u, long long n, double *d_jp2, double *d_fjp,
                              double *d_p2, double *d_plen, ReduceBuf rb, cudaStream_t st) {
  OpLineSearchIn op{jp, f, p, u, {d_jp2, d_fjp, d_p2, d_plen}};
  reduce_multi(op, n, rb, st);
}
void launch_step_norms(const double *f, long long n, double *d_f2, double *d_fmax, ReduceBuf rb,
                       cudaStream_t st) {
  OpStepNorms op{f, {d_f2, d_fmax}};
  reduce_multi(op, n, rb, st);
}
void launch_init_norms(const double *u, const double *f, long long n, double *d_u2,
                       double *d_fmax, double *d_f2, ReduceBuf rb, cudaStream_t st) {
  OpInitNorms op{u, f, {d_u2, d_fmax, d_f2}};
  reduce_multi(op, n, rb, st);
}

// ---- difference-quotient J v (kinspgmr.c:481-518, uscale = 1) ---------------
// d[0..2] = <u, v>, <v, v>, |v|_1 from OpDQ; writes sigma to d[3] and 1/sigma
// to d[4]: sigma = sign(<u, v>) sqrt_relfunc max(|<u, v>|, |v|_1) / <v, v>
__global__ void k_dq_sigma(double *d, double sqrt_relfunc) {
  pdl_enter();
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    const double sutsv = d[0], vtv = d[1], sq1norm = d[2];
    const double sign = (sutsv >= 0.0) ? 1.0 : -1.0;
    const double a = fabs(sutsv);
    const double sigma = sign * sqrt_relfunc * (a > sq1norm ? a : sq1norm) / vtv;
    d[3] = sigma;
    d[4] = 1.0 / sigma;
  }
}
// w = sigma v + u
__global__ void k_dq_point(double *__restrict__ w, const double *__restrict__ u,
                           const double *__restrict__ v, const double *__restrict__ d,
                           long long n) {
  pdl_enter();
  const double sigma = d[3];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    w[i] = sigma * v[i] + u[i];
}
// z = (1/sigma) (fw - f)
__global__ void k_dq_finish(double *__restrict__ z, const double *__restrict__ fw,
                            const double *__restrict__ f, const double *__restrict__ d,
                            long long n) {
  pdl_enter();
  const double sigma_inv = d[4];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    z[i] = sigma_inv * (fw[i] - f[i]);
}
static inline int grid_for(long long n);
void launch_dq_prepare(const double *u, const double *v, long long n, double *d,
                       double sqrt_relfunc, ReduceBuf rb, cudaStream_t st) {
  OpDQ op{u, v, {d, d + 1, d + 2}};
  reduce_multi(op, n, rb, st);
  launch_pdl(k_dq_sigma, dim3(1), dim3(32), st, d, sqrt_relfunc);
}
void launch_dq_point(double *w, const double *u, const double *v, const double *d, long long n,
                     cudaStream_t st) {
  launch_pdl(k_dq_point, dim3(grid_for(n)), dim3(256), st, w, u, v, d, n);
}
void launch_dq_finish(double *z, const double *fw, const double *f, const double *d,
                      long long n, cudaStream_t st) {
  launch_pdl(k_dq_finish, dim3(grid_for(n)), dim3(256), st, z, fw, f, d, n);
}

// ---- element-wise ---------------------------------------------------------
__global__ void k_axpby(double *__restrict__ y, const double *__restrict__ x, double a, double b,
                        long long n) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    y[i] = (b == 0.0) ? a * x[i] : a * x[i] + b * y[i];
}
__global__ void k_xpay(double *__restrict__ z, const double *__restrict__ x, double a,
                       const double *__restrict__ y, long long n) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    z[i] = x[i] + a * y[i];
}
__global__ void k_scale_inv_dev(double *__restrict__ x, const double *__restrict__ s,
                                long long n) {
  pdl_enter();
  double a = 1.0 / (*s);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] *= a;
}
__global__ void k_scale(double *__restrict__ x, double a, long long n) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] *= a;
}
__global__ void k_fill(double *__restrict__ x, double v, long long n) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] = v;
}
struct VecList {
  const double *v[NK_MAX_KRYLOV + 1];
};
// xcor = yg[0] V0 + 0, then xcor = yg[k] Vk + xcor (sequential N_VLinearSum order)
// xcor = sum_k yg[k] V_k, accumulated in k order onto 0 (accumulate = 0) or
// onto xcor itself (accumulate = 1: a GMRES restart cycle adds to the
// correction of the earlier cycles, spgmr.c:357-358)
__global__ void k_combine(double *__restrict__ xcor, VecList V, const double *__restrict__ yg,
                          int kdim, long long n, int accumulate) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double acc = accumulate ? xcor[i] : 0.0;
    for (int k = 0; k < kdim; k++) acc = yg[k] * V.v[k][i] + 1.0 * acc;
    xcor[i] = acc;
  }
}

// restart direction V_0 = yg[0] V_0 + sum_{k=1..kdim} yg[k] V_k, in place
// (spgmr.c:405-409): every element reads only its own index
__global__ void k_restart_v0(double *v0, VecList V, const double *__restrict__ yg, int kdim,
                             long long n) {
  pdl_enter();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double acc = yg[0] * v0[i];
    for (int k = 1; k <= kdim; k++) acc = yg[k] * V.v[k][i] + 1.0 * acc;
    v0[i] = acc;
  }
}

static inline int grid_for(long long n) {
  long long b = (n + 255) / 256;
  return (int)(b < 148 * 16 ? (b < 1 ? 1 : b) : 148 * 16);
}

void launch_axpby(double *y, const double *x, double a, double b, long long n, cudaStream_t st) {
  launch_pdl(k_axpby, dim3(grid_for(n)), dim3(256), st, y, x, a, b, n);
}
void launch_xpay(double *z, const double *x, double a, const double *y, long long n,
                 cudaStream_t st) {
  launch_pdl(k_xpay, dim3(grid_for(n)), dim3(256), st, z, x, a, y, n);
}
void launch_scale_inv_dev(double *x, const double *s, long long n, cudaStream_t st) {
  launch_pdl(k_scale_inv_dev, dim3(grid_for(n)), dim3(256), st, x, s, n);
}
void launch_scale(double *x, double a, long long n, cudaStream_t st) {
  launch_pdl(k_scale, dim3(grid_for(n)), dim3(256), st, x, a, n);
}
void launch_fill(double *x, double v, long long n, cudaStream_t st) {
  launch_pdl(k_fill, dim3(grid_for(n)), dim3(256), st, x, v, n);
}
void launch_combine(double *xcor, double *const *V, const double *yg, int kdim, long long n,
                    cudaStream_t st, int accumulate) {
  VecList L;
  for (int k = 0; k < kdim && k <= NK_MAX_KRYLOV; k++) L.v[k] = V[k];
  launch_pdl(k_combine, dim3(grid_for(n)), dim3(256), st, xcor, L, yg, kdim, n, accumulate);
}
void launch_restart_v0(double *const *V, const double *yg, int kdim, long long n,
                       cudaStream_t st) {
  VecList L;
  for (int k = 0; k <= kdim && k <= NK_MAX_KRYLOV; k++) L.v[k] = V[k];
  launch_pdl(k_restart_v0, dim3(grid_for(n)), dim3(256), st, V[0], L, yg, kdim, n);
}

// ---- the same steps with their scalars on the device (graph solve) ---------
// V0 of a GMRES cycle: b / ||b|| = src * (bsign / r_norm) on the first cycle
// (as launch_axpby with b = 0), the restart direction / its norm after
__global__ void k_v0_init(double *__restrict__ v0, const double *__restrict__ src,
                          const NkState *S, const double *__restrict__ sc, long long n) {
  pdl_enter();
  const bool first = S->ntries == 0;
  const double a = first ? S->k.bsign * (1.0 / S->r_norm) : 1.0 / sc[SCI_RNORM];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    if (first)
      v0[i] = a * src[i];
    else
      v0[i] *= a;
  }
}
__global__ void k_combine_dev(double *__restrict__ xcor, VecList V, const double *__restrict__ yg,
                              const int *kdim_p, const int *acc_p, long long n) {
  pdl_enter();
  const int kdim = *kdim_p, accumulate = *acc_p;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double acc = accumulate ? xcor[i] : 0.0;
    for (int k = 0; k < kdim; k++) acc = yg[k] * V.v[k][i] + 1.0 * acc;
    xcor[i] = acc;
  }
}
__global__ void k_restart_v0_dev(double *v0, VecList V, const double *__restrict__ yg,
                                 const int *kdim_p, long long n) {
  pdl_enter();
  const int kdim = *kdim_p;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    double acc = yg[0] * v0[i];
    for (int k = 1; k <= kdim; k++) acc = yg[k] * V.v[k][i] + 1.0 * acc;
    v0[i] = acc;
  }
}
__global__ void k_scale_inv_dev_unless(double *__restrict__ x, const double *__restrict__ s,
                                       const int *skip, long long n) {
  pdl_enter();
  if (*skip) return;
  double a = 1.0 / (*s);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] *= a;
}
__global__ void k_fill_if(double *__restrict__ x, double v, const int *flag, long long n) {
  pdl_enter();
  if (!*flag) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] = v;
}
__global__ void k_scale_if(double *__restrict__ x, const double *a_p, const int *flag,
                           long long n) {
  pdl_enter();
  if (!*flag) return;
  const double a = *a_p;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    x[i] *= a;
}
__global__ void k_copy_if(double *__restrict__ dst, const double *__restrict__ src,
                          const int *flag, long long n) {
  pdl_enter();
  if (!*flag) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

void launch_v0_init(double *v0, const double *src, const NkState *S, const double *sc,
                    long long n, cudaStream_t st) {
  launch_pdl(k_v0_init, dim3(grid_for(n)), dim3(256), st, v0, src, S, sc, n);
}
void launch_combine_dev(double *xcor, double *const *V, int nv, const double *yg, const int *kdim,
                        const int *accumulate, long long n, cudaStream_t st) {
  VecList L{};
  for (int k = 0; k < nv && k <= NK_MAX_KRYLOV; k++) L.v[k] = V[k];
  launch_pdl(k_combine_dev, dim3(grid_for(n)), dim3(256), st, xcor, L, yg, kdim, accumulate, n);
}
void launch_restart_v0_dev(double *const *V, int nv, const double *yg, const int *kdim,
                           long long n, cudaStream_t st) {
  VecList L{};
  for (int k = 0; k < nv && k <= NK_MAX_KRYLOV; k++) L.v[k] = V[k];
  launch_pdl(k_restart_v0_dev, dim3(grid_for(n)), dim3(256), st, V[0], L, yg, kdim, n);
}
void launch_scale_inv_dev_unless(double *x, const double *s, const int *skip, long long n,
                                 cudaStream_t st) {
  launch_pdl(k_scale_inv_dev_unless, dim3(grid_for(n)), dim3(256), st, x, s, skip, n);
}
void launch_fill_if(double *x, double v, const int *flag, long long n, cudaStream_t st) {
  launch_pdl(k_fill_if, dim3(grid_for(n)), dim3(256), st, x, v, flag, n);
}
void launch_scale_if(double *x, const double *a, const int *flag, long long n, cudaStream_t st) {
  launch_pdl(k_scale_if, dim3(grid_for(n)), dim3(256), st, x, a, flag, n);
}
void launch_copy_if(double *dst, const double *src, const int *flag, long long n,
                    cudaStream_t st) {
  launch_pdl(k_copy_if, dim3(grid_for(n)), dim3(256), st, dst, src, flag, n);
}

// ---- GMRES scalars ----------------------------------------------------------
// S layout: [0, (lmax+1)*lmax) Hessenberg H(i,j) at i*lmax+j; then givens
// (2*lmax), yg (lmax+1), then named scalars.
struct GS {
  double *H, *giv, *yg, *sc;
  int lmax;
  __device__ double &h(int i, int j) { return H[i * lmax + j]; }
};
enum { SC_RNORM = 0, SC_ROT, SC_RHO, SC_VKNORM2, SC_NEWNORM2, SC_HLL, SC_BETA, SC_QRFAIL };

__device__ GS gs_view(double *S, int lmax) {
  GS g;
  g.lmax = lmax;
  g.H = S;
  g.giv = S + (lmax + 1) * lmax;
  g.yg = g.giv + 2 * lmax;
  g.sc = g.yg + lmax + 1;
  return g;
}

__device__ void givens(double t1, double t2, double &c, double &s) {
  if (t2 == 0.0) {
    c = 1.0;
    s = 0.0;
  } else if (fabs(t2) >= fabs(t1)) {
    double t3 = t1 / t2;
    s = -1.0 / sqrt(1.0 + t3 * t3);
    c = -s * t3;
  } else {
    double t3 = t2 / t1;
    c = 1.0 / sqrt(1.0 + t3 * t3);
    s = -c * t3;
  }
}

__device__ __forceinline__ void gmres_scalar_op(int op, double *S, int l, int lmax) {
  GS g = gs_view(S, lmax);
  double *sc = g.sc;
  switch (op) {
    case 0: {  // start: r_norm = sqrt(<V0,V0>) already in SC_RNORM as squared
      for (int i = threadIdx.x; i < (lmax + 1) * lmax; i += blockDim.x) g.H[i] = 0.0;
      if (threadIdx.x != 0) break;
      double r = sqrt(sc[SC_RNORM]);
      sc[SC_RNORM] = r;
      sc[SC_BETA] = r;
      sc[SC_ROT] = 1.0;
      sc[SC_RHO] = r;
      break;
    }
    case 4: {  // QRsol with krydim = l (iterativ.c:253-286)
      int kd = l;
      g.yg[0] = sc[SC_RNORM];
      for (int i = 1; i <= kd; i++) g.yg[i] = 0.0;
      for (int k = 0; k < kd; k++) {
        double c = g.giv[2 * k], s = g.giv[2 * k + 1];
        double t1 = g.yg[k], t2 = g.yg[k + 1];
        g.yg[k] = c * t1 - s * t2;
        g.yg[k + 1] = s * t1 + c * t2;
      }
      sc[SC_QRFAIL] = 0.0;
      for (int k = kd - 1; k >= 0; k--) {
        if (g.h(k, k) == 0.0) {
          sc[SC_QRFAIL] = 1.0;
          break;
        }
        g.yg[k] /= g.h(k, k);
        for (int i = 0; i < k; i++) g.yg[i] -= g.yg[k] * g.h(i, k);
      }
      break;
    }
    case 6: {  // restart (spgmr.c:390-404), krydim = l: the residual direction's
               // coefficients yg and the new r_norm
      int kd = l;
      double s_product = 1.0;
      for (int i = kd; i > 0; i--) {
        g.yg[i] = s_product * g.giv[2 * i - 2];
        s_product *= g.giv[2 * i - 1];
      }
      g.yg[0] = s_product;
      double r_norm = sc[SC_RNORM] * s_product;
      for (int i = 0; i <= kd; i++) g.yg[i] *= r_norm;
      sc[SC_RNORM] = fabs(r_norm);
      break;
    }
    case 7: {  // next restart cycle: Hessenberg cleared, rotation product 1
      for (int i = threadIdx.x; i < (lmax + 1) * lmax; i += blockDim.x) g.H[i] = 0.0;
      if (threadIdx.x == 0) sc[SC_ROT] = 1.0;
      break;
    }
  }
}
__global__ void k_gmres_scalar(int op, double *S, int l, int lmax) {
  pdl_enter();
  gmres_scalar_op(op, S, l, lmax);
}
// the same step with its column / Krylov dimension read from the device
__global__ void k_gmres_scalar_dev(int op, double *S, const int *l, int lmax) {
  pdl_enter();
  gmres_scalar_op(op, S, *l, lmax);
}

// Scalar end of GMRES iteration l (one thread): column l of the Hessenberg
// matrix in h[0 .. l + 1], h[l + 1] the norm of the new vector; the rotations
// of the earlier columns in giv.  The Givens update and the residual estimate
// (iterativ.c:205-250) and, St given, the control step that arms the next
// iteration (spgmr.c:340-360).
__device__ __forceinline__ void gmres_column(const GS &g, double *h, const double *giv, int l,
                                             NkState *St, const NkConds &C) {
  double *sc = g.sc;
  const int k = l + 1;
  for (int i = 0; i < l; i++) {
    const double t1 = h[i], t2 = h[i + 1], c = giv[2 * i], s = giv[2 * i + 1];
    h[i] = c * t1 - s * t2;
    h[i + 1] = s * t1 + c * t2;
  }
  double c, s;
  const double t1 = h[l], t2 = h[k];
  givens(t1, t2, c, s);
  h[l] = c * t1 - s * t2;
  g.giv[2 * l] = c;
  g.giv[2 * l + 1] = s;
  for (int i = 0; i <= k; i++) g.H[i * g.lmax + k - 1] = h[i];
  const double rot = sc[SC_ROT] * s, rho = fabs(rot * sc[SC_RNORM]);
  sc[SC_ROT] = rot;
  sc[SC_RHO] = rho;
  sc[SC_HLL] = t2;
  if (St) {
    St->execs[NKB_GM0 + l]++;
    St->lin_iters++;
    St->pc_solves++;
    if (St->k.use_dq) St->fevals++;
    St->krydim = l + 1;
    St->rho = rho;
    if (rho <= St->delta)
      St->converged = 1;
    else if (l + 1 < St->k.lmax)
      cudaGraphSetConditional(C.iter[l + 1], 1u);
  }
}
// ModifiedGS's test whether the projections cancelled the vector (iterativ.c:60-66)
__device__ __forceinline__ bool cancelled(double vk_norm, double new_norm) {
  const double temp = 1000.0 * vk_norm;
  return !((temp + new_norm) != temp);
}
// its second pass (iterativ.c:68-84): one product against basis vector i
__device__ __forceinline__ bool reorth_step(double np, double &hi, double &nn2) {
  const double temp = 1000.0 * hi;
  if ((temp + np) == temp) return false;
  hi += np;
  nn2 += np * np;
  return true;
}
__device__ __forceinline__ double reorth_norm(double hk, double nn2) {
  const double np2 = hk * hk - nn2;
  return (np2 > 0.0) ? sqrt(np2) : 0.0;
}

// Re-orthogonalisation of a long vector over the whole grid, as phases: phase p
// takes product p - 1 off vk and sums its product with V[p], in chunks (items)
// that any block may claim; the block that finishes a phase's last item adds the
// partial sums in item order, takes ModifiedGS's decision (reorth_step) and
// lets the next phase begin.  No block waits for one that is not running: an
// unfinished item belongs to a block that has claimed it, so the launch needs
// no co-residency.  Waits are bounded; a block that gives up writes 4 into the
// error word and leaves.
struct ReorthCtl {  // behind the scalars of S; zero between launches
  unsigned next[NK_MAX_KRYLOV + 1], done[NK_MAX_KRYLOV + 1], ready[NK_MAX_KRYLOV + 1], left;
  double coef[NK_MAX_KRYLOV + 1], nn2;
};
static_assert(sizeof(ReorthCtl) <= GS_REORTH_DOUBLES * sizeof(double), "its space in S");
constexpr int FIN_THREADS = 512;
constexpr unsigned long long FIN_WAIT_NS = 1000000000ull;  // 1 s

__device__ __forceinline__ double block_sum(double a, double *red) {
  const int t = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) a = a + __shfl_down_sync(0xffffffffu, a, o);
  if ((t & 31) == 0) red[t >> 5] = a;
  __syncthreads();
  a = red[0];
  for (int w = 1; w < FIN_THREADS / 32; w++) a = a + red[w];
  __syncthreads();  // (red may be written again)
  return a;
}

// true in the one block that leaves last, when everything is done
__device__ bool reorthogonalise(const VecList &V, double *vk, long long n, unsigned items,
                                long long chunk, double *partial, const GS &g, int k,
                                ReorthCtl *ctl, int *kerr) {
  const int t = threadIdx.x;
  __shared__ double red[FIN_THREADS / 32], coef;
  __shared__ unsigned word;
  __shared__ bool gave_up;
  for (int p = 0; p <= k; p++) {
    double a = 0.0;  // coefficient of V[p - 1]
    if (p > 0) {
      if (t == 0) {
        gave_up = false;
        unsigned long long since = 0;
        for (unsigned it = 1; ld_acquire_gpu(&ctl->ready[p - 1]) == 0; it++) {
          __nanosleep(64);
          if (it % 64) continue;
          const unsigned long long now = global_ns();
          if (!since) since = now;
          if (now - since > FIN_WAIT_NS || *(volatile int *)kerr) {
            *(volatile int *)kerr = 4;
            gave_up = true;
            break;
          }
        }
        coef = __ldcg(&ctl->coef[p - 1]);
      }
      __syncthreads();
      if (gave_up) break;
      a = coef;
    }
    if (p == k && a == 0.0) break;
    const double *x = p > 0 ? V.v[p - 1] : nullptr, *z = p < k ? V.v[p] : nullptr;
    for (;;) {
      __syncthreads();
      if (t == 0) word = atomicAdd(&ctl->next[p], 1u);
      __syncthreads();
      const unsigned item = word;
      if (item >= items) break;
      const long long q0 = item * chunk, q1 = min(n, q0 + chunk);
      double acc = 0.0;
#pragma unroll 4
      for (long long q = q0 + t; q < q1; q += FIN_THREADS) {
        double y = __ldcg(vk + q);  // (another block's store of the phase before)
        if (a != 0.0) {
          y = y + a * x[q];
          __stcg(vk + q, y);
        }
        if (z) acc = acc + z[q] * y;
      }
      const double sum = block_sum(acc, red);
      if (t == 0) {
        __stcg(partial + item, sum);
        word = atom_add_acq_rel_gpu(&ctl->done[p], 1u);
      }
      __syncthreads();
      if (word + 1 != items || !z) continue;
      // the phase's last item
      acc = 0.0;
      for (unsigned q = t; q < items; q += FIN_THREADS) acc = acc + __ldcg(partial + q);
      const double np = block_sum(acc, red);
      if (t == 0) {
        double *hp = g.H + p * g.lmax + k - 1, h = __ldcg(hp), nn2 = __ldcg(&ctl->nn2);
        const bool apply = reorth_step(np, h, nn2);
        __stcg(hp, h);
        __stcg(&ctl->nn2, nn2);
        __stcg(&ctl->coef[p], apply ? -np : 0.0);
        atom_add_acq_rel_gpu(&ctl->ready[p], 1u);
      }
    }
  }
  __syncthreads();
  if (t == 0) word = atom_add_acq_rel_gpu(&ctl->left, 1u);
  __syncthreads();
  return word + 1 == gridDim.x;
}

// End of GMRES iteration l in one launch, the projections and their dot
// products done: one block stages a few scalars in shared memory and does them,
// the others leave at once, unless ModifiedGS re-orthogonalises (iterativ.c:60-84),
// which is for a new vector that lost all but 1e-13 of its norm: an exact
// breakdown.  It stands for 3 l + 7 launches of 1.5 to 3 us each, most of
// them gated off.
__global__ void __launch_bounds__(FIN_THREADS) k_gmres_finish(
    VecList V, double *vk, long long n, unsigned items, long long chunk, double *partial,
    double *S, int l, int lmax, NkState *St, NkConds C, int *kerr) {
  const GS g = gs_view(S, lmax);
  const double *sc = g.sc;
  const int k = l + 1, t = threadIdx.x;
  __shared__ double h[NK_MAX_KRYLOV + 1], giv[2 * NK_MAX_KRYLOV];
  if (t < 2 * l) giv[t] = g.giv[t];  // (older than the kernel before this one)
  pdl_enter();
  // (the column is asked for together with the norms: one round trip)
  const double *column = g.H + t * lmax + k - 1;
  double ht = t < k ? __ldcg(column) : 0.0;
  double hk = sqrt(sc[SC_NEWNORM2]);
  if (cancelled(sqrt(sc[SC_VKNORM2]), hk)) {
    ReorthCtl *ctl = reinterpret_cast<ReorthCtl *>(g.sc + SCI_COUNT);
    if (!reorthogonalise(V, vk, n, items, chunk, partial, g, k, ctl, kerr)) return;
    const double nn2 = __ldcg(&ctl->nn2);
    if (nn2 != 0.0) hk = reorth_norm(hk, nn2);
    if (*(volatile int *)kerr) hk = nan("");
    if (t < k) ht = __ldcg(column);
    __syncthreads();
    for (int q = t; q < (int)(sizeof(ReorthCtl) / 4); q += FIN_THREADS)
      reinterpret_cast<unsigned *>(ctl)[q] = 0u;
  } else if (blockIdx.x != 0) {
    return;
  }
  if (t < k) h[t] = ht;
  __syncthreads();
  if (t != 0) return;
  h[k] = hk;
  gmres_column(g, h, giv, l, St, C);
}

// The whole end of GMRES iteration l on one thread-block cluster, for vectors
// that fit its registers' reach: modified Gram-Schmidt (iterativ.c:30-86) of
// V[l + 1] against V[0 .. l], re-orthogonalisation, and the column's scalars.
// The new vector stays in shared memory; a dot product is a block reduction and
// one exchange of the blocks' partial sums through distributed shared memory
// (added in block order, so every block holds the same bits).  It stands for
// l + 3 launches with a grid-wide reduction each.
// A timestep of 12x10x8 in FP64: 1.25 ms against 1.36.  Up to 65536 cells: at
// 131072 (16384 per block) it is no faster than the launches, whose passes the
// whole GPU streams.
constexpr int MGS_THREADS = 1024, MGS_CLUSTER = 8, MGS_CELLS = 8 * 1024;  // cells per block
struct MgsCluster {
  double *sh;               // block reduction
  double (*part)[2][MGS_CLUSTER];  // [step parity][value][block]
  int step, rank, blocks;
  // sums over the cluster of a (and b)
  __device__ __forceinline__ void sum(double &a, double &b, bool both) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a = a + __shfl_down_sync(0xffffffffu, a, o);
      if (both) b = b + __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      sh[w] = a;
      if (both) sh[32 + w] = b;
    }
    __syncthreads();
    double (*dst)[MGS_CLUSTER] = part[step & 1];
    if (w < (both ? 2 : 1)) {
      double v = sh[32 * w + lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, o);
      v = __shfl_sync(0xffffffffu, v, 0);
      if (lane < blocks) {  // to every block
        const uint32_t mine = (uint32_t)__cvta_generic_to_shared(&dst[w][rank]);
        uint32_t at;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(mine), "r"(lane));
        asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(at), "d"(v) : "memory");
      }
    }
    if (blocks > 1) {
      asm volatile("barrier.cluster.arrive.release;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else {
      __syncthreads();
    }
    a = dst[0][0];
    for (int q = 1; q < blocks; q++) a = a + dst[0][q];
    if (both) {
      b = dst[1][0];
      for (int q = 1; q < blocks; q++) b = b + dst[1][q];
    }
    step++;
  }
};
__global__ void __launch_bounds__(MGS_THREADS, 1) k_gmres_mgs(VecList V, double *vk, int n,
                                                              double *S, int l, int lmax,
                                                              NkState *St, NkConds C) {
  extern __shared__ double own[];  // this block's cells of vk
  __shared__ double sh[64], h[NK_MAX_KRYLOV + 1], giv[2 * NK_MAX_KRYLOV], part[2][2][MGS_CLUSTER];
  const int t = threadIdx.x, k = l + 1;
  unsigned rank, blocks;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(blocks));
  MgsCluster R{sh, part, 0, (int)rank, (int)blocks};
  const GS g = gs_view(S, lmax);
  if (t < 2 * l) giv[t] = g.giv[t];  // (older than the kernel before this one)
  const int per = (n + (int)blocks - 1) / (int)blocks, c0 = (int)rank * per;
  const int m = min(per, n - c0);  // cells of this block (none: n < c0)
  // a block's shared memory is written by the others from their first sum on
  if (blocks > 1) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
  pdl_enter();
  const double *src = vk + c0, *v0 = V.v[0] + c0;
  double a = 0.0, b = 0.0;
#pragma unroll 4
  for (int q = t; q < m; q += MGS_THREADS) {
    const double y = src[q];
    own[q] = y;
    a = a + y * y;
    b = b + v0[q] * y;
  }
  R.sum(a, b, true);
  const double vk_norm = sqrt(a);
  double hi = b;
  for (int i = 0; i < k; i++) {
    if (t == 0) h[i] = hi;
    const double *x = V.v[i] + c0, *z = i + 1 < k ? V.v[i + 1] + c0 : nullptr;
    const double w = -1.0 * hi;
    a = 0.0;
#pragma unroll 4
    for (int q = t; q < m; q += MGS_THREADS) {
      const double y = own[q] + w * x[q];
      own[q] = y;
      a = a + (z ? z[q] : y) * y;
    }
    R.sum(a, b, false);
    hi = a;
  }
  double hk = sqrt(hi), nn2 = 0.0;
  if (cancelled(vk_norm, hk)) {
    for (int i = 0; i < k; i++) {
      const double *x = V.v[i] + c0;
      a = 0.0;
      for (int q = t; q < m; q += MGS_THREADS) a = a + x[q] * own[q];
      R.sum(a, b, false);
      // (every thread of the cluster decides alike, on the same h)
      double hq = h[i];
      const bool apply = reorth_step(a, hq, nn2);
      __syncthreads();
      if (t == 0) h[i] = hq;
      if (apply)
        for (int q = t; q < m; q += MGS_THREADS) own[q] = own[q] - a * x[q];
      __syncthreads();
    }
    if (nn2 != 0.0) hk = reorth_norm(hk, nn2);
  }
  double *dst = vk + c0;
  for (int q = t; q < m; q += MGS_THREADS) dst[q] = own[q];
  if (t == 0 && rank == 0) {
    h[k] = hk;
    gmres_column(g, h, giv, l, St, C);
  }
  // no block leaves while another may still write its partial sums
  if (blocks > 1) {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
  }
}
cudaError_t krylov_prepare_kernels() {
  return cudaFuncSetAttribute(k_gmres_mgs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              MGS_CELLS * (int)sizeof(double));
}

// Whether launch_gmres_mgs takes vectors of n elements
bool gmres_mgs_fits(long long n) {
  static const long long most = [] {
    const char *v = getenv("PFGPU_MGS_CELLS");
    const long long all = (long long)MGS_CLUSTER * MGS_CELLS;
    const long long m = v && *v ? atoll(v) : all;
    return m < all ? m : all;
  }();
  return n <= most;
}
void launch_gmres_mgs(double *const *V, int l, int lmax, long long n, double *S, cudaStream_t st,
                      NkState *St, const NkConds *C) {
  VecList L{};
  for (int k = 0; k <= l; k++) L.v[k] = V[k];
  int blocks = 1;
  while (blocks < MGS_CLUSTER && (long long)blocks * 2 * MGS_THREADS < n) blocks *= 2;
  const size_t smem = (size_t)((n + blocks - 1) / blocks) * sizeof(double);
  launch_pdl_cluster(k_gmres_mgs, blocks, dim3(MGS_THREADS), smem, st, L, V[l + 1], (int)n, S, l,
                     lmax, St, C ? *C : NkConds{});
}

void launch_gmres_finish(double *const *V, int l, int lmax, long long n, double *S,
                         double *partial, int *kerr, cudaStream_t st, NkState *St, const NkConds *C) {
  VecList L{};
  for (int k = 0; k <= l; k++) L.v[k] = V[k];
  // a block per SM and two chunks for each, of 2048 cells (whole lines) and more
  long long items = (n + 2047) / 2048;
  if (items > 2 * 148) items = 2 * 148;
  if (items < 1) items = 1;
  const long long chunk = ((n + items - 1) / items + 15) / 16 * 16;
  items = (n + chunk - 1) / chunk;
  launch_pdl(k_gmres_finish, dim3((unsigned)((items + 1) / 2)), dim3(FIN_THREADS), st, L, V[l + 1],
             n, (unsigned)items, chunk, partial, S, l, lmax, St, C ? *C : NkConds{}, kerr);
}

void launch_gmres_scalar(int op, double *S, int l, int lmax, cudaStream_t st) {
  // (the two that clear the Hessenberg matrix: a thread per entry)
  const int threads = op == GM_START || op == GM_RESTART_INIT ? 256 : 1;
  launch_pdl(k_gmres_scalar, dim3(1), dim3(threads), st, op, S, l, lmax);
}
void launch_gmres_scalar_dev(int op, double *S, const int *l, int lmax, cudaStream_t st) {
  launch_pdl(k_gmres_scalar_dev, dim3(1), dim3(1), st, op, S, l, lmax);
}
// ---- ParFlow layout <-> dense ------------------------------------------------
__global__ void k_unpad(const double *__restrict__ pad, double *__restrict__ dense, int nx,
                        int ny, int nz) {
  pdl_enter();
  long long n = (long long)nx * ny * nz;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
       c += (long long)gridDim.x * blockDim.x) {
    int i = (int)(c % nx);
    long long r = c / nx;
    int j = (int)(r % ny), k = (int)(r / ny);
    dense[c] = pad[(i + 1) + (long long)(nx + 2) * ((j + 1) + (long long)(ny + 2) * (k + 1))];
  }
}
__global__ void k_pad(const double *__restrict__ dense, double *__restrict__ pad, int nx, int ny,
                      int nz) {
  pdl_enter();
  long long n = (long long)(nx + 2) * (ny + 2) * (nz + 2);
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
       c += (long long)gridDim.x * blockDim.x) {
    int i = (int)(c % (nx + 2)) - 1;
    long long r = c / (nx + 2);
    int j = (int)(r % (ny + 2)) - 1, k = (int)(r / (ny + 2)) - 1;
    bool in = i >= 0 && j >= 0 && k >= 0 && i < nx && j < ny && k < nz;
    pad[c] = in ? dense[i + (long long)nx * (j + (long long)ny * k)] : 0.0;
  }
}
// dense -> a frame of g ghost layers on every side (ghosts written as 0)
__global__ void k_pad_ghost(const double *__restrict__ dense, double *__restrict__ pad, int nx,
                            int ny, int nz, int g) {
  pdl_enter();
  const int px = nx + 2 * g, py = ny + 2 * g;
  long long n = (long long)px * py * (nz + 2 * g);
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n;
       c += (long long)gridDim.x * blockDim.x) {
    int i = (int)(c % px) - g;
    long long r = c / px;
    int j = (int)(r % py) - g, k = (int)(r / py) - g;
    bool in = i >= 0 && j >= 0 && k >= 0 && i < nx && j < ny && k < nz;
    pad[c] = in ? dense[i + (long long)nx * (j + (long long)ny * k)] : 0.0;
  }
}
void launch_pad_ghost(const double *dense, double *pad, int nx, int ny, int nz, int g,
                      cudaStream_t st) {
  const long long n = (long long)(nx + 2 * g) * (ny + 2 * g) * (nz + 2 * g);
  launch_pdl(k_pad_ghost, dim3(grid_for(n)), dim3(256), st, dense, pad, nx, ny, nz, g);
}
void launch_unpad(const double *pad, double *dense, int nx, int ny, int nz, cudaStream_t st) {
  launch_pdl(k_unpad, dim3(grid_for((long long)nx * ny * nz)), dim3(256), st, pad, dense, nx, ny, nz);
}
void launch_pad(const double *dense, double *pad, int nx, int ny, int nz, cudaStream_t st) {
  launch_pdl(k_pad, dim3(grid_for((long long)(nx + 2) * (ny + 2) * (nz + 2))), dim3(256), st, dense, pad, nx, ny,
                                                                             nz);
}

}  // namespace pfgpu
