// The coarse tail of a V-cycle with a red/black smoother: every level of at
// most 1024 cells (PFGPU_TAIL_CELLS) in one thread block, out of shared memory.
//
// What bounds it: nothing but the chain of dependent phases.  The tail holds
// about eleven levels and each passes through eight phases that need one
// another's values, most of them on a single warp, whose dependent
// instructions issue one per four cycles or more.  So the kernel is built for
// few instructions between one phase and the next:
//  * everything that does not depend on the iterate is worked out once per
//    multigrid setup (k_tail_pack) and copied in as it lies: the operator by
//    rows, the transfer weights by cell, a record of indices per pair of
//    cells.  The copy runs ahead of the wait on the preceding kernel;
//  * a thread owns one pair of cells (2q, 2q+1) of a row, one of each colour,
//    and keeps both rows in registers for a whole leg of a level; the rows of
//    the next level are loaded while the current one finishes;
//  * the iterate has a frame of zero ghosts, so a sweep is six loads and a
//    multiply-add chain without a test;
//  * the restriction reads only the colour that was not swept last, and the
//    thread that restricts to a coarse pair starts that pair's zero-guess red
//    sweep at once;
//  * a phase waits only on the warps that hold cells of its level: named
//    barriers over power-of-two groups of warps, __syncwarp once one warp is
//    enough (levels of at most 64 cells, half of all levels).
// The generic tail (k_vcycle_tail_smem: nine barriers of 1024 threads per level,
// two level descriptors copied per thread and leg) took 85 us in FP64 and 83 us
// with the scaled FP16 operator at 512x512x50; this one takes 23.5 and 23 us.
// V-cycle graph of a 12x10x8 grid, all tail: 43 us against 103.
// Spreading levels of up to 8192 cells over a cluster of eight blocks (iterate
// in distributed shared memory) did not pay: a phase cost 2000 cycles there
// (470 of them the release / acquire barrier of 512-thread blocks, the rest
// remote loads), as much as a launch of its own.
#include <cstdint>
#include <type_traits>

#include "mg_common.cuh"
#include "pdl.cuh"
#include "pfgpu_kernels.h"

namespace pfgpu {
namespace {

constexpr int NTH = 512;                 // threads, one per pair of the first level
constexpr size_t SMEM_MAX = 220 * 1024;  // dynamic shared memory

// Pair record.  Bits: F0 = 1 << 28, F1 = 1 << 29.
struct __align__(16) Rec {
  int x;   // framed index of the even cell | red slot * F0 | second cell exists * F1
  int c;   // its linear index
  int up;  // framed index of the coarse point at / below the black cell | fine point * F0 |
           // coarse point above * F1
  int dn;  // finer level: linear index of the point under the even cell | flags << 24: computed
           // (bit 0), lower (1), upper (2) neighbour exists; the same for the odd cell (3 .. 5)
};
constexpr int IDX = (1 << 28) - 1, IDX24 = (1 << 24) - 1;

template <typename T>
struct alignas(16) Row {
  T v[8];  // w e s n l u, the diagonal, the right-hand side
};
template <typename T>
struct Wt {
  T w1, w2;
};

struct TailLevel {
  int nx, ny, nz, dir;
  int n, np, warps;     // cells, pairs, warps that hold the pairs (a power of two)
  int o_x;              // byte offsets in shared memory: framed iterate
  int o_row, o_w, o_r;  // rows, weights, records (also, less o_img, in the packed image)
};
struct TailPlan {
  int nt;
  int nonsym;          // red, black (else red, black, red)
  int o_t;             // residual (scratch of the level in progress)
  int o_img, img;      // the packed image in shared memory, its bytes
  void *image;         // ... and in global memory
  const void *b;
  void *x;
  const int *hflag;
  TailLevel L[TAIL_MAX_LEVELS];
};
// sources of the packing
struct TailSrc {
  const void *op[TAIL_MAX_LEVELS][4], *w1[TAIL_MAX_LEVELS], *w2[TAIL_MAX_LEVELS];
};
static_assert(sizeof(TailPlan) + sizeof(TailSrc) <= 4000, "they are kernel parameters");

__device__ __forceinline__ int frame_px(const TailLevel &L) { return L.nx + 1; }
__device__ __forceinline__ int frame_sz(const TailLevel &L) { return (L.nx + 1) * (L.ny + 1); }
// one ghost column and row (each the upper ghost of one line and the lower
// ghost of the next), a ghost plane at either end
__device__ __forceinline__ int framed(const TailLevel &L, int i, int j, int k) {
  return i + (L.nx + 1) * (j + (L.ny + 1) * (k + 1));
}

__device__ __forceinline__ float to_t(const __half *p, float) { return __half2float(*p); }
template <typename T>
__device__ __forceinline__ T to_t(const T *p, T) {
  return *p;
}

// Fills the image after a setup: thread e < cells the row and weights of one
// cell of one level, the threads after them the record of one pair.
template <typename T, bool H>
__global__ void __launch_bounds__(128) k_tail_pack(const __grid_constant__ TailPlan P,
                                                   const __grid_constant__ TailSrc S, int cells) {
  pdl_enter();
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned char *img = reinterpret_cast<unsigned char *>(P.image) - P.o_img;
  const int nt = P.nt;
  int l = 0;
  if (e < cells) {
    for (; e >= P.L[l].n; l++) e -= P.L[l].n;
    const TailLevel &L = P.L[l];
    const int c = e, nx = L.nx, sz = L.nx * L.ny;
    const int i = c % nx, j = c / nx % L.ny, k = c / sz;
    using O = typename std::conditional<H, __half, T>::type;
    const O *oe = reinterpret_cast<const O *>(S.op[l][0]),
            *on = reinterpret_cast<const O *>(S.op[l][1]),
            *ou = reinterpret_cast<const O *>(S.op[l][2]),
            *od = reinterpret_cast<const O *>(S.op[l][3]);
    Row<T> r;
    r.v[0] = i > 0 ? to_t(oe + c - 1, T(0)) : T(0);
    r.v[1] = to_t(oe + c, T(0));
    r.v[2] = j > 0 ? to_t(on + c - nx, T(0)) : T(0);
    r.v[3] = to_t(on + c, T(0));
    r.v[4] = k > 0 ? to_t(ou + c - sz, T(0)) : T(0);
    r.v[5] = to_t(ou + c, T(0));
    r.v[6] = to_t(od + c, T(0));
    r.v[7] = T(0);
    reinterpret_cast<Row<T> *>(img + L.o_row)[c] = r;
    if (l + 1 < nt)
      reinterpret_cast<Wt<T> *>(img + L.o_w)[c] =
          Wt<T>{reinterpret_cast<const T *>(S.w1[l])[c], reinterpret_cast<const T *>(S.w2[l])[c]};
    return;
  }
  e -= cells;
  for (; l < nt && e >= P.L[l].np; l++) e -= P.L[l].np;
  if (l >= nt) return;
  const TailLevel &L = P.L[l];
  const int hx = (L.nx + 1) >> 1, i0 = 2 * (e % hx), j = e / hx % L.ny, k = e / (hx * L.ny);
  const int r = (j + k) & 1;  // parity of the even cell: 1 means it is red
  Rec q;
  q.x = framed(L, i0, j, k) | (r ^ 1) << 28 | (i0 + 1 < L.nx) << 29;
  q.c = i0 + L.nx * (j + L.ny * k);
  q.up = q.dn = 0;
  if (l + 1 < nt) {
    const TailLevel &C = P.L[l + 1];
    const int D = L.dir, ox = D == 0, oy = D == 1, oz = D == 2, bi = i0 + r;
    const int cd = D == 0 ? bi : D == 1 ? j : k, nd = D == 0 ? L.nx : D == 1 ? L.ny : L.nz;
    if (bi < L.nx)
      q.up = framed(C, bi >> ox, j >> oy, k >> oz) | (cd & 1) << 28 |
             ((cd & 1) && cd + 1 < nd) << 29;
  }
  if (l > 0) {
    const TailLevel &F = P.L[l - 1];
    const int D = F.dir, ox = D == 0, oy = D == 1, oz = D == 2;
    const int zpar = P.nonsym ? 0 : 1;  // parity of the colour swept last
    const int fi0 = i0 << ox, fj = j << oy, fk = k << oz;
    q.dn = fi0 + F.nx * (fj + F.ny * fk);
    for (int s = 0; s < 2; s++) {
      const int fi = fi0 + (s << ox);
      const int cd = D == 0 ? fi : D == 1 ? fj : fk, nd = D == 0 ? F.nx : D == 1 ? F.ny : F.nz;
      const int comp = ((fi + fj + fk) & 1) != zpar;
      q.dn |= (comp | (cd > 0) << 1 | (cd + 1 < nd) << 2) << (24 + 3 * s);
    }
  }
  reinterpret_cast<Rec *>(img + L.o_r)[e] = q;
}

// barrier over the first `warps` warps (a power of two)
__device__ __forceinline__ void group_sync(int warps) {
  if (warps == 1) {
    __syncwarp();
  } else {
    const int id = 32 - __clz(warps);  // 2 .. 5
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(warps * 32) : "memory");
  }
}

// restriction of the finer level's residual t to the coarse point over fine
// point f (bits: computed, lower, upper)
template <typename T, bool H>
__device__ __forceinline__ T restrict_small(const T *t, const Wt<T> *w, int f, int so, int bits) {
  const bool comp = bits & 1, lo = bits & 2, hi = bits & 4;
  const T rc = comp ? t[f] : T(0);
  const T rm = !comp && lo ? t[f - so] : T(0), rp = !comp && hi ? t[f + so] : T(0);
  return restrict_value<T, H>(H ? w[f].w1 : T(0), rc, lo ? w[f - so].w2 : T(0), rm,
                              hi ? w[f + so].w1 : T(0), rp);
}

// a thread's pair on one level: its rows and where its cells live
template <typename T>
struct Pair {
  Row<T> red, black;
  Rec q;
  __device__ bool has_red() const { return (q.x >> 28 & 1) == 0 || (q.x >> 29 & 1); }
  __device__ bool has_black() const { return (q.x >> 28 & 1) || (q.x >> 29 & 1); }
  __device__ int rs() const { return q.x >> 28 & 1; }
  __device__ void load(const TailLevel &L, const unsigned char *sm) {
    if ((int)threadIdx.x < L.np) {
      q = reinterpret_cast<const Rec *>(sm + L.o_r)[threadIdx.x];
      const Row<T> *row = reinterpret_cast<const Row<T> *>(sm + L.o_row) + q.c;
      if (has_red()) red = row[rs()];
      if (has_black()) black = row[rs() ^ 1];
    } else {
      q.x = -1;  // (never used: guarded by act)
    }
  }
};

template <typename T, bool H>
__global__ void __launch_bounds__(NTH, 1) k_tail(const __grid_constant__ TailPlan P) {
  extern __shared__ __align__(16) unsigned char sm[];
  // the level table in shared memory: indexed reads of the parameter would go
  // through the constant cache, a miss per level
  __shared__ TailLevel V[TAIL_MAX_LEVELS];
  const int th = threadIdx.x, warp = th >> 5, nt = P.nt;
  // Neither the image nor the flag is written by the kernel before this one
  // (the setup lies further back), so they are read ahead of the wait.
  {
    const char *src = reinterpret_cast<const char *>(P.image);
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(sm + P.o_img);
    for (int o = th * 16; o < P.img; o += NTH * 16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + o), "l"(src + o)
                   : "memory");
  }
  for (int e = th; e < nt * (int)(sizeof(TailLevel) / 4); e += NTH)
    reinterpret_cast<uint32_t *>(V)[e] = reinterpret_cast<const uint32_t *>(P.L)[e];
  for (int e = th; e < P.o_t / 16; e += NTH)  // iterates and their ghosts
    reinterpret_cast<uint4 *>(sm)[e] = make_uint4(0, 0, 0, 0);
  const bool u = H && *P.hflag == 0;  // unit diagonal
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  T *tt = reinterpret_cast<T *>(sm + P.o_t);
  // Gauss-Seidel update of the cell at x (rb_update's operations and order)
  auto relax = [&](const Row<T> &r, T *x, int px, int sz) {
    const T xw = x[-1], xe = x[1], xs = x[-px], xn = x[px], xl = x[-sz], xu = x[sz];
    if (u) {
      T acc = mul_rn(r.v[0], xw);
      acc = fma(r.v[1], xe, acc);
      acc = fma(r.v[2], xs, acc);
      acc = fma(r.v[3], xn, acc);
      acc = fma(r.v[4], xl, acc);
      acc = fma(r.v[5], xu, acc);
      *x = r.v[7] - acc;
    } else {
      *x = rb_update<T>(r.v[6], r.v[7], r.v[0], xw, r.v[1], xe, r.v[2], xs, r.v[3], xn, r.v[4],
                        xl, r.v[5], xu);
    }
  };
  Pair<T> A;
  A.load(V[0], sm);
  pdl_enter();
  if (th < V[0].np) {
    const T *gb = reinterpret_cast<const T *>(P.b) + A.q.c;
    Row<T> *row = reinterpret_cast<Row<T> *>(sm + V[0].o_row) + A.q.c;
    const int rs = A.rs();
    if (A.has_red()) row[rs].v[7] = A.red.v[7] = gb[rs];
    if (A.has_black()) row[rs ^ 1].v[7] = A.black.v[7] = gb[rs ^ 1];
  }
  int low = -1;  // coarsest level this warp takes part in
  // down
  for (int l = 0; l < nt; l++) {
    const TailLevel &L = V[l];
    const int W = L.warps;
    if (warp >= W) break;
    low = l;
    const bool act = th < L.np, coarsest = l + 1 == nt;
    const int px = frame_px(L), sz = frame_sz(L);
    const bool hr = act && A.has_red(), hb = act && A.has_black();
    const int rs = A.rs();
    T *x = reinterpret_cast<T *>(sm + L.o_x) + (A.q.x & IDX);
    T *xr = x + rs, *xb = x + (rs ^ 1);
    if (l > 0 && act) {
      Row<T> *row = reinterpret_cast<Row<T> *>(sm + L.o_row) + A.q.c;
      const TailLevel &F = V[l - 1];
      const Wt<T> *w = reinterpret_cast<const Wt<T> *>(sm + F.o_w);
      const int D = F.dir, so = D == 0 ? 1 : D == 1 ? F.nx : F.nx * F.ny, f = A.q.dn & IDX24;
      const int step = D == 0 ? 2 : 1;
      if (hr) {
        A.red.v[7] = restrict_small<T, H>(tt, w, f + rs * step, so, A.q.dn >> (24 + 3 * rs));
        row[rs].v[7] = A.red.v[7];
      }
      if (hb) {
        A.black.v[7] =
            restrict_small<T, H>(tt, w, f + (rs ^ 1) * step, so, A.q.dn >> (24 + 3 * (rs ^ 1)));
        row[rs ^ 1].v[7] = A.black.v[7];
      }
    }
    // zero-guess red sweep
    if (hr) *xr = u ? A.red.v[7] : A.red.v[7] / A.red.v[6];
    group_sync(W);
    if (hb) relax(A.black, xb, px, sz);
    group_sync(W);
    if (!P.nonsym || coarsest) {  // the coarse solve is red, black, red
      if (hr) relax(A.red, xr, px, sz);
      if (coarsest) break;
      group_sync(W);
    }
    // residual of the colour not swept last
    if (P.nonsym ? hr : hb) {
      const Row<T> &r = P.nonsym ? A.red : A.black;
      const T *p = P.nonsym ? xr : xb;
      tt[A.q.c + (P.nonsym ? rs : rs ^ 1)] = residual_value<T>(
          r.v[7], u ? T(1) : r.v[6], *p, r.v[0], p[-1], r.v[1], p[1], r.v[2], p[-px], r.v[3],
          p[px], r.v[4], p[-sz], r.v[5], p[sz]);
    }
    if (warp < V[l + 1].warps) A.load(V[l + 1], sm);
    group_sync(W);
  }
  // up
  if (low >= 0 && low + 1 == nt) low--;
  if (low >= 0) A.load(V[low], sm);
  for (int l = low; l >= 0; l--) {
    const TailLevel &L = V[l], &C = V[l + 1];
    const int W = L.warps;
    const bool act = th < L.np;
    const int px = frame_px(L), sz = frame_sz(L);
    const bool hr = act && A.has_red(), hb = act && A.has_black();
    const int rs = A.rs();
    T *x = reinterpret_cast<T *>(sm + L.o_x) + (A.q.x & IDX);
    T *xr = x + rs, *xb = x + (rs ^ 1);
    Wt<T> w{T(0), T(0)};
    const T *xc = reinterpret_cast<const T *>(sm + C.o_x) + (A.q.up & IDX);
    if (hb) w = reinterpret_cast<const Wt<T> *>(sm + L.o_w)[A.q.c + (rs ^ 1)];
    const int D = L.dir, so = D == 0 ? 1 : D == 1 ? frame_px(C) : frame_sz(C);
    group_sync(W);  // the coarse level is done
    if (hb) {
      const T el = xc[0], eh = A.q.up >> 29 & 1 ? xc[so] : T(0);
      *xb = add_rn(*xb, prolong_value<T, H>(A.q.up >> 28 & 1, w.w1, w.w2, el, eh));
    }
    group_sync(W);
    if (hr) relax(A.red, xr, px, sz);
    group_sync(W);
    if (hb) relax(A.black, xb, px, sz);
    if (!P.nonsym) {
      group_sync(W);
      if (hr) relax(A.red, xr, px, sz);
    }
    if (l > 0) A.load(V[l - 1], sm);
  }
  // the first level's iterate back
  __syncthreads();
  if (th < V[0].np) {
    const Rec q = reinterpret_cast<const Rec *>(sm + V[0].o_r)[th];
    const T *x = reinterpret_cast<const T *>(sm + V[0].o_x) + (q.x & IDX);
    T *gx = reinterpret_cast<T *>(P.x) + q.c;
    gx[0] = x[0];
    if (q.x >> 29 & 1) gx[1] = x[1];
  }
}

long long pad16b(long long bytes) { return (bytes + 15) / 16 * 16; }

// plan of the levels first .. nl-1; its shared-memory bytes, or -1 when they
// do not fit (more pairs than threads, or the shared memory)
template <typename T>
long long tail_layout(const MGLevel<T> *L, int first, int nl, bool h16, TailPlan *P, TailSrc *S) {
  const long long ts = sizeof(T);
  *P = TailPlan{};
  if (S) *S = TailSrc{};
  P->nt = nl - first;
  if (P->nt > TAIL_MAX_LEVELS) return -1;
  long long o = 0;
  for (int q = 0; q < P->nt; q++) {
    const MGLevel<T> &M = L[first + q];
    const long long np = (long long)((M.nx + 1) / 2) * M.ny * M.nz;
    if (np > NTH) return -1;
    TailLevel &D = P->L[q];
    D.nx = M.nx; D.ny = M.ny; D.nz = M.nz;
    D.dir = M.dir;
    D.n = (int)M.n;
    D.np = (int)np;
    D.warps = 1;
    while (32 * D.warps < np) D.warps *= 2;
    D.o_x = (int)o;
    o += pad16b((M.nx + 1LL) * (M.ny + 1LL) * (M.nz + 2LL) * ts);
    if (o > (long long)SMEM_MAX) return -1;
    if (S) {
      for (int s = 0; s < 4; s++)  // E N U, then the diagonal
        S->op[q][s] = h16 ? (const void *)M.h[s] : (const void *)M.a[(s + 1) & 3];
      S->w1[q] = h16 ? M.q1 : M.p1;
      S->w2[q] = h16 ? M.q2 : M.p2;
    }
  }
  P->o_t = (int)o;
  o += pad16b(P->L[0].n * ts);
  P->o_img = (int)o;
  for (int q = 0; q < P->nt; q++) {
    TailLevel &D = P->L[q];
    D.o_row = (int)o;
    o += 8LL * D.n * ts;
    D.o_w = (int)o;
    if (q + 1 < P->nt) o = pad16b(o + 2LL * D.n * ts);
    D.o_r = (int)o;
    o += 16LL * D.np;
    if (o > (long long)SMEM_MAX) return -1;
  }
  P->img = (int)o - P->o_img;
  return o;
}

}  // namespace

template <typename T>
size_t tail_image_bytes(const MGLevel<T> *L, int first, int nl, bool h16) {
  TailPlan P;
  return tail_layout(L, first, nl, h16, &P, nullptr) < 0 ? 0 : (size_t)P.img;
}

template <typename T>
cudaError_t tail_pairs_prepare() {
  cudaError_t e = cudaFuncSetAttribute(k_tail<T, false>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
  if constexpr (std::is_same<T, float>::value)
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_tail<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)SMEM_MAX);
  return e;
}

template <typename T>
void launch_tail_pack(const MGLevel<T> *L, int first, int nl, int smoother, void *image,
                      cudaStream_t st, bool h16) {
  TailPlan P;
  TailSrc S;
  tail_layout(L, first, nl, h16, &P, &S);
  P.nonsym = smoother == 2;
  P.image = image;
  int cells = 0, pairs = 0;
  for (int q = 0; q < P.nt; q++) {
    cells += P.L[q].n;
    pairs += P.L[q].np;
  }
  const dim3 grid((cells + pairs + 127) / 128);
  if constexpr (std::is_same<T, float>::value) {
    if (h16) {
      launch_pdl(k_tail_pack<T, true>, grid, dim3(128), st, P, S, cells);
      return;
    }
  }
  launch_pdl(k_tail_pack<T, false>, grid, dim3(128), st, P, S, cells);
}

template <typename T>
void launch_tail_pairs(const MGLevel<T> *L, int first, int nl, int smoother, void *image,
                       cudaStream_t st, bool h16, const T *b, T *x) {
  TailPlan P;
  const size_t smem = (size_t)tail_layout(L, first, nl, h16, &P, nullptr);
  P.nonsym = smoother == 2;
  P.image = image;
  P.b = b ? b : L[first].b;
  P.x = x ? x : L[first].x;
  P.hflag = L[first].hflag;
  if constexpr (std::is_same<T, float>::value) {
    if (h16) {
      launch_pdl_smem(k_tail<T, true>, dim3(1), dim3(NTH), smem, st, P);
      return;
    }
  }
  launch_pdl_smem(k_tail<T, false>, dim3(1), dim3(NTH), smem, st, P);
}

#define INST(T)                                                                              \
  template size_t tail_image_bytes<T>(const MGLevel<T> *, int, int, bool);                   \
  template cudaError_t tail_pairs_prepare<T>();                                              \
  template void launch_tail_pack<T>(const MGLevel<T> *, int, int, int, void *, cudaStream_t, \
                                    bool);                                                   \
  template void launch_tail_pairs<T>(const MGLevel<T> *, int, int, int, void *, cudaStream_t, \
                                     bool, const T *, T *);
INST(double)
INST(float)

}  // namespace pfgpu
