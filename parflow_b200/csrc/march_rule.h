// Which of their two launch forms the residual and the Jacobian take (host
// code, no CUDA): gather, a thread per cell, or march, a warp per 31 columns of
// a row that walks up a chunk of planes.  Both give the same bits.
//
// Both are bound by instruction issue, so they cost by the lanes they launch,
// cells or not: a row takes 32 ceil(nx / 31) in the march form and bx
// ceil(nx / bx) in the gather form.  Per lane march is the cheaper one (four
// faces instead of six), the more so the more waves of warps a launch holds.
// Measured (us, march / gather; heterogeneous K, unsaturated, each with its van
// Genuchten pass), with r = march's lanes over gather's:
//   residual        r 0.75  80x150x50 27.4 / 27.9, 80x250x50 37.5 / 46.0
//                   r 1     96x125x50 27.6 / 25.7, 62x323x50 37.7 / 40.8
//                   r 1.25  128x94x50 27.4 / 24.8, 128x469x50 108 / 117
//                   r 1.5   64x313x50 47.8 / 40.1, 64x938x50 118 / 117
//                   r 2     32x625x50 52.0 / 42.2, 32x1875x50 142 / 123
//   ... with slopes r 1.5   64x188x50 33.7 / 38.6;  r 2  32x625x50 64.1 / 60.7
//   Jacobian, FP32  r 1.25  128x391x12 30.3 / 30.4, 128x469x50 125 / 148
//                   r 1.5   64x188x50 36.2 / 30.7, 64x938x50 138 / 148
//                   r 2     32x625x50 60.0 / 50.3, 32x1875x50 165 / 148
//   Jacobian, FP64  r 1     62x807x12 30.2 / 36.9, 96x521x12 40.5 / 36.3
//                   r 1.5   64x782x12 39.2 / 34.7, 64x938x50 169 / 166
// 96x521x12: at three blocks per SM a grid just above one wave (528 blocks of
// 444) leaves the second nearly empty, unless its blocks are those of a short
// last chunk (48x250x50, 448 blocks of which the last hold two planes:
// 34.5 / 40.8).
#pragma once

namespace pfgpu {

constexpr int MARCH_WARPS = 8, MARCH_COLS = 31;
constexpr long long MARCH_MIN_CELLS = 600000;

// columns of a gather block of `threads` threads
inline int gather_columns(int nx, int threads) {
  int bx = 32;
  while (bx < nx && bx < 128) bx *= 2;
  return bx < threads ? bx : threads;
}

// planes per chunk of a march: about eight or more (each chunk costs one more z
// face per column), four waves of 32 warps per SM where the planes allow it
inline int march_planes(int nx, int ny, int nz) {
  const long long strips = (long long)((nx + MARCH_COLS - 1) / MARCH_COLS) * ny;
  const long long want = 4LL * 32 * 148, most = (nz + 7) / 8;
  long long chunks = (want + strips - 1) / strips;
  if (chunks > most) chunks = most;
  return (int)((nz + chunks - 1) / chunks);
}

enum MarchKernel { MARCH_RESIDUAL, MARCH_JACOBIAN_F32, MARCH_JACOBIAN_F64 };

// (slopes: terrain-following or overland; FP64 Jacobians take gather there:
// 128x157x50 75.3 / 70.5 with march, 256x196x12 50.1 / 46.1)
inline bool march_pays(MarchKernel kernel, bool slopes, int nx, int ny, int nz) {
  if ((long long)nx * ny * nz < MARCH_MIN_CELLS) return false;
  if (kernel == MARCH_JACOBIAN_F64 && slopes) return false;
  const int bx = gather_columns(nx, kernel == MARCH_RESIDUAL ? 256 : 128);
  const long long strips = (nx + MARCH_COLS - 1) / MARCH_COLS, row = (nx + bx - 1LL) / bx * bx;
  const double lanes = (double)row * ny * nz, r = 32.0 * (double)strips / (double)row;
  if (r >= 1.75) return false;
  if (kernel == MARCH_RESIDUAL) return slopes || lanes >= 700e3 * r * r;
  if (r >= 1.3 && lanes < 2e6) return false;
  if (kernel == MARCH_JACOBIAN_F64 || slopes) {  // three blocks per SM
    const int planes = march_planes(nx, ny, nz), chunks = (nz + planes - 1) / planes;
    const long long wave = 3 * 148,
                    blocks = strips * ((ny + MARCH_WARPS - 1) / MARCH_WARPS) * chunks;
    const bool short_last = 2 * (nz - (chunks - 1) * planes) <= planes;
    if (blocks > wave && 5 * blocks < 6 * wave && !short_last) return false;
  }
  return true;
}

}  // namespace pfgpu
