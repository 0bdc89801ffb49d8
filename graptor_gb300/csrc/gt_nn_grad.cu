// Parameter gradients of the warm-start network's convolutions (sm_103a).
//
// Weight gradient: dW[co][ci][t] = sum over batch and voxels of dY[co][v] X[ci][v + off(t)], dY
// in float32.  It is bound by FP32 multiply-adds once its operands come from shared
// memory: a block stages a tile of X with its halo and of dY, and a thread keeps all 27
// taps of one input and two output channels in registers while it slides along a row: a
// voxel costs 9 + 1 shared-memory loads (11 of the 128-byte write-backs) for 54 multiply-adds.
// Staging is what is left over: a block's tiles follow each other in depth, so that a tile
// stages one new plane of three, its loads are all in flight before the first is stored, and
// two blocks per SM stage and multiply in turn.  (Four output channels per thread need fewer
// loads, 13 for 108, but 226 registers, one block per SM: 268 us for 16 x 16 channels on
// 4 x 16 x 64 x 64 voxels.  The form before, a 16 x 64 tile GEMM that gathered every tap's operand
// from global memory, took 1010 us there and 3010 us for 48 x 16;
// this one 116 and 314 us.)
//
// Sums are deterministic: a block adds its tiles in order and writes one partial sum per
// weight, a second kernel adds the blocks' partial sums in a fixed order.
#include <cooperative_groups.h>

#include "graptor_gb300.h"
#include "gt_nn.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int WG_C = 16;   // input and output channels of a block
constexpr int WG_V = 128;  // voxels of a tile: HR rows of WB

template <int HR, int WB>
struct WTile {
  static constexpr int XS = WG_C + 1, YS = WG_C + 2;  // channel strides (bank conflicts of the staging)
  float dy[HR][WB][YS];
  float x[3][HR + 2][WB + 2][XS];  // planes d - 1, d, d + 1, each at its depth modulo 3
};

// 256 threads: two groups of 128 (each half of a tile's rows), thread = (input channel, pair
// of output channels).  Block (ci tile, co tile, slot) sums tiles [slot * per, (slot + 1) * per).
template <class TX, int HR, int WB>
__global__ void __launch_bounds__(256, 2) k_wgrad3(const float *__restrict__ dy, int Co, int Cdy, int dy_off,
                                                   const TX *__restrict__ x, int Ci, int Cx, int x_off, Shape s,
                                                   int tiles, int per, float *__restrict__ part) {
  static_assert(HR * WB == WG_V && HR % 2 == 0 && (WB == 16 || WB == 32), "tile shape");
  extern __shared__ float4 smem4[];
  WTile<HR, WB> &T = *reinterpret_cast<WTile<HR, WB> *>(smem4);
  constexpr int XS = WTile<HR, WB>::XS, XR = (WB + 2) * XS;
  const int ci0 = blockIdx.x * WG_C, co0 = blockIdx.y * WG_C;
  const int group = threadIdx.x >> 7, ci = threadIdx.x & 15, cp = (threadIdx.x >> 4) & 7;
  const int nw = (s.W + WB - 1) / WB, nh = (s.H + HR - 1) / HR;
  const long long vol = (long long)s.H * s.W * s.D;
  float acc[2][27];
#pragma unroll
  for (int t = 0; t < 27; ++t) acc[0][t] = acc[1][t] = 0.f;
  const int t0 = blockIdx.z * per, t1 = min(tiles, t0 + per);
  for (int t = t0; t < t1; ++t) {
    int r = t;
    const int d = r % s.D; r /= s.D;
    const int w0 = (r % nw) * WB; r /= nw;
    const int h0 = (r % nh) * HR;
    const int b = r / nh;
    // a staging thread's column is fixed, its rows and channels step through the tile
    const int lw = threadIdx.x % WB, lq = threadIdx.x / WB;
    constexpr int STEP = 256 / WB;
    float gq[WG_V * WG_C / 256];
    {
      const float *p = dy + ((long long)b * Cdy + dy_off + co0) * vol + ((long long)d * s.H + h0) * s.W + w0 + lw;
#pragma unroll
      for (int k = 0; k < WG_V * WG_C / 256; ++k) {
        const int q = lq + k * STEP, c = q / HR, hr = q % HR;
        gq[k] = (co0 + c < Co && h0 + hr < s.H && w0 + lw < s.W) ? __ldg(p + c * vol + hr * s.W) : 0.f;
      }
    }
    __syncthreads();  // the tile before has been used
#pragma unroll
    for (int k = 0; k < WG_V * WG_C / 256; ++k) {
      const int q = lq + k * STEP;
      T.dy[q % HR][lw][q / HR] = gq[k];
    }
    // planes: all three at the start of a column, the next one after that
    for (int zd = (t == t0 || d == 0) ? d - 1 : d + 1; zd <= d + 1; ++zd) {
      float(*X)[WB + 2][XS] = T.x[(zd + 3) % 3];
      const bool in_d = zd >= 0 && zd < s.D;
      const TX *p = x + ((long long)b * Cx + x_off + ci0) * vol + ((long long)zd * s.H + h0 - 1) * s.W + w0;
      constexpr int ROWS = (HR + 2) * WG_C, NK = ROWS / STEP;
      static_assert(ROWS % STEP == 0 && 2 * ROWS <= 2 * 256, "staging");
      float v[NK], e[2];
      auto in_row = [&](int q) {
        const int zh = h0 + q % (HR + 2) - 1;
        return in_d && ci0 + q / (HR + 2) < Ci && zh >= 0 && zh < s.H;
      };
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int q = lq + k * STEP;
        v[k] = (in_row(q) && w0 + lw < s.W) ? ld<TX>(p + (q / (HR + 2)) * vol + (q % (HR + 2)) * s.W + lw) : 0.f;
      }
      // the columns beside the tile: (row, side) pairs
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int m = threadIdx.x + 256 * k, q = m >> 1, zw = w0 + ((m & 1) ? WB : -1);
        e[k] = (m < 2 * ROWS && in_row(q) && zw >= 0 && zw < s.W)
                   ? ld<TX>(p + (q / (HR + 2)) * vol + (q % (HR + 2)) * s.W + zw - w0) : 0.f;
      }
#pragma unroll
      for (int k = 0; k < NK; ++k) {
        const int q = lq + k * STEP;
        X[q % (HR + 2)][1 + lw][q / (HR + 2)] = v[k];
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int m = threadIdx.x + 256 * k, q = m >> 1;
        if (m < 2 * ROWS) X[q % (HR + 2)][(m & 1) ? WB + 1 : 0][q / (HR + 2)] = e[k];
      }
    }
    __syncthreads();
    const float *rows[3] = {&T.x[(d + 2) % 3][0][0][ci], &T.x[d % 3][0][0][ci], &T.x[(d + 1) % 3][0][0][ci]};
    // Only the tile's voxels inside the volume: the others' dY is 0, but 0 times an infinite X
    // would be NaN.
    const int hv = min(HR, s.H - h0), wv = min(WB, s.W - w0);
#pragma unroll 1
    for (int hr = group * (HR / 2); hr < min((group + 1) * (HR / 2), hv); ++hr) {
      float win[9][3];  // X at (kd, kh) and three neighbours along the row
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        win[k][1] = rows[k / 3][(hr + k % 3) * XR];
        win[k][2] = rows[k / 3][(hr + k % 3) * XR + XS];
      }
      auto voxel = [&](int ww) {
        const float2 g = *reinterpret_cast<const float2 *>(&T.dy[hr][ww][2 * cp]);
#pragma unroll
        for (int k = 0; k < 9; ++k) {
          win[k][0] = win[k][1];
          win[k][1] = win[k][2];
          win[k][2] = rows[k / 3][(hr + k % 3) * XR + (ww + 2) * XS];
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            acc[0][3 * k + q] = fmaf(g.x, win[k][q], acc[0][3 * k + q]);
            acc[1][3 * k + q] = fmaf(g.y, win[k][q], acc[1][3 * k + q]);
          }
        }
      };
      if (wv == WB) {
#pragma unroll
        for (int ww = 0; ww < WB; ++ww) voxel(ww);
      } else {
#pragma unroll 1
        for (int ww = 0; ww < wv; ++ww) voxel(ww);
      }
    }
  }
  // the second group's sums are added to the first's, one output channel of the pair at a time
  float *red = reinterpret_cast<float *>(smem4);
#pragma unroll
  for (int o = 0; o < 2; ++o) {
    __syncthreads();
    if (group == 1) {
#pragma unroll
      for (int t = 0; t < 27; ++t) red[t * 128 + (threadIdx.x & 127)] = acc[o][t];
    }
    __syncthreads();
    if (group == 0 && ci0 + ci < Ci && co0 + 2 * cp + o < Co) {
      float *p = part + (((size_t)blockIdx.z * Co + co0 + 2 * cp + o) * Ci + ci0 + ci) * 27;
#pragma unroll
      for (int t = 0; t < 27; ++t) p[t] = acc[o][t] + red[t * 128 + threadIdx.x];
    }
  }
}

// 1x1x1 kernels: a thread sums its voxels for 4 output and 8 input channels, the block adds its
// threads in a fixed order.  Block (ci tile, co tile, slot) takes voxels [slot * per, ...).
constexpr int W1_O = 4, W1_I = 8;

template <class TX>
__global__ void __launch_bounds__(256) k_wgrad1(const float *__restrict__ dy, int Co, int Cdy, int dy_off,
                                                const TX *__restrict__ x, int Ci, int Cx, int x_off, long long vol,
                                                long long nvox, long long per, float *__restrict__ part) {
  __shared__ float sh[8][W1_O * W1_I];
  const int ci0 = blockIdx.x * W1_I, co0 = blockIdx.y * W1_O;
  float acc[W1_O][W1_I];
#pragma unroll
  for (int o = 0; o < W1_O; ++o)
#pragma unroll
    for (int c = 0; c < W1_I; ++c) acc[o][c] = 0.f;
  const long long v1 = min(nvox, (long long)(blockIdx.z + 1) * per);
  for (long long v = (long long)blockIdx.z * per + threadIdx.x; v < v1; v += 256) {
    const long long b = v / vol, rv = v - b * vol;
    float g[W1_O], a[W1_I];
#pragma unroll
    for (int o = 0; o < W1_O; ++o) g[o] = co0 + o < Co ? dy[((size_t)b * Cdy + dy_off + co0 + o) * vol + rv] : 0.f;
#pragma unroll
    for (int c = 0; c < W1_I; ++c) a[c] = ci0 + c < Ci ? ld<TX>(x + ((size_t)b * Cx + x_off + ci0 + c) * vol + rv) : 0.f;
#pragma unroll
    for (int o = 0; o < W1_O; ++o)
#pragma unroll
      for (int c = 0; c < W1_I; ++c) acc[o][c] = fmaf(g[o], a[c], acc[o][c]);
  }
#pragma unroll
  for (int o = 0; o < W1_O; ++o)
#pragma unroll
    for (int c = 0; c < W1_I; ++c) {
      float r = acc[o][c];
#pragma unroll
      for (int k = 16; k > 0; k >>= 1) r += __shfl_xor_sync(0xffffffffu, r, k);
      if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5][o * W1_I + c] = r;
    }
  __syncthreads();
  if (threadIdx.x < W1_O * W1_I) {
    const int o = threadIdx.x / W1_I, c = threadIdx.x - o * W1_I;
    float r = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) r += sh[k][threadIdx.x];
    if (co0 + o < Co && ci0 + c < Ci) part[((size_t)blockIdx.z * Co + co0 + o) * Ci + ci0 + c] = r;
  }
}

// g (+)= sum of the slots' partial sums: a block adds 32 weights, 8 warps each every eighth
// slot, then the warps in order
__global__ void __launch_bounds__(256) k_wgrad_reduce(const float *__restrict__ part, int nslot, long long n,
                                                      float *__restrict__ g, int accumulate) {
  __shared__ float sh[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long t = (long long)blockIdx.x * 32 + lane;
  float a = 0.f;
  if (t < n) {
#pragma unroll 4
    for (int c = warp; c < nslot; c += 8) a += part[(size_t)c * n + t];
  }
  sh[warp][lane] = a;
  __syncthreads();
  if (warp == 0 && t < n) {
    float r = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) r += sh[k][lane];
    g[t] = accumulate ? g[t] + r : r;
  }
}

// db[co] (+)= sum over batch and voxels of dY: a cluster of 8 blocks per channel, each an
// eighth of the voxels, added in a fixed order through distributed shared memory.  HBM bound; one
// block per channel (16 blocks on 152 SMs) took 229 us for 16 x 262144 values.  Up to 2048 values of
// a channel one block: the cluster's barriers cost more (64 x 1024 values 5.1 us, 3.8 with one block).
constexpr int BG_CL = 8;
constexpr long long BG_ONE = 2048;

template <int CL>
__global__ void __cluster_dims__(CL, 1, 1) __launch_bounds__(256)
    k_bias_grad(const float *__restrict__ dy, int Cdy, int dy_off, long long vol, int B, int vec,
                float *__restrict__ db, int accumulate) {
  __shared__ float sh[8];
  __shared__ float total;
  const int co = blockIdx.x / CL, rank = blockIdx.x % CL;
  float a = 0.f;
  for (int b = 0; b < B; ++b) {
    const float *__restrict__ p = dy + ((size_t)b * Cdy + dy_off + co) * vol;
    if (vec) {  // vol a multiple of 4, dy on a 16-byte boundary
      for (long long v = rank * 256 + threadIdx.x; v < vol / 4; v += CL * 256) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(p) + v);
        a += (q.x + q.y) + (q.z + q.w);
      }
    } else {
      for (long long v = rank * 256 + threadIdx.x; v < vol; v += CL * 256) a += p[v];
    }
  }
#pragma unroll
  for (int k = 16; k > 0; k >>= 1) a += __shfl_xor_sync(0xffffffffu, a, k);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
  __syncthreads();
  if (threadIdx.x == 0) {
    float r = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) r += sh[k];
    total = r;
    if (CL == 1) db[co] = accumulate ? db[co] + r : r;
  }
  if constexpr (CL == 1) return;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  if (rank == 0 && threadIdx.x == 0) {
    float r = 0.f;
#pragma unroll
    for (int k = 0; k < CL; ++k) r += *cl.map_shared_rank(&total, k);
    db[co] = accumulate ? db[co] + r : r;
  }
  cl.sync();  // the other blocks' shared memory is read until here
}

template <class TX, int HR, int WB>
cudaError_t wgrad3(const float *dy, int Co, int Cdy, int dy_off, const void *x, int Ci, int Cx, int x_off, Shape s,
                   long long nchunk, float *part, int *nslot, cudaStream_t st) {
  const long long tiles = (long long)s.B * s.D * ((s.H + HR - 1) / HR) * ((s.W + WB - 1) / WB);
  if (tiles > (1ll << 30)) return cudaErrorInvalidValue;
  const long long per = (tiles + nchunk - 1) / nchunk;
  *nslot = (int)((tiles + per - 1) / per);
  auto kern = k_wgrad3<TX, HR, WB>;
  const int smem = (int)sizeof(WTile<HR, WB>);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid(nblk(Ci, WG_C), nblk(Co, WG_C), (unsigned)*nslot);
  kern<<<grid, 256, smem, st>>>(dy, Co, Cdy, dy_off, (const TX *)x, Ci, Cx, x_off, s, (int)tiles, (int)per, part);
  return cudaGetLastError();
}

template <class TX>
cudaError_t wgrad(int ks, const float *dy, int Co, int Cdy, int dy_off, const void *x, int Ci, int Cx, int x_off,
                  Shape s, long long nchunk, float *part, int *nslot, cudaStream_t st) {
  if (ks == 3) {
    // rows of 32 voxels where they are filled, of 16 otherwise
    if (s.W % 32 == 0 || s.W > 64)
      return wgrad3<TX, 4, 32>(dy, Co, Cdy, dy_off, x, Ci, Cx, x_off, s, nchunk, part, nslot, st);
    return wgrad3<TX, 8, 16>(dy, Co, Cdy, dy_off, x, Ci, Cx, x_off, s, nchunk, part, nslot, st);
  }
  const long long vol = (long long)s.D * s.H * s.W, nvox = vol * s.B;
  const long long per = (nvox + nchunk - 1) / nchunk;
  *nslot = (int)((nvox + per - 1) / per);
  const dim3 grid(nblk(Ci, W1_I), nblk(Co, W1_O), (unsigned)*nslot);
  k_wgrad1<TX><<<grid, 256, 0, st>>>(dy, Co, Cdy, dy_off, (const TX *)x, Ci, Cx, x_off, vol, nvox, per, part);
  return cudaGetLastError();
}

}  // namespace

extern "C" {

// part must hold nchunk * Co * Ci * K3 floats; nchunk = ceil(voxels / kchunk) bounds the number
// of blocks per channel tile (and of partial sums)
int gt_nn_conv3d_wgrad(const float *dy, int Co, int Cdy, int dy_off, const void *x, int x_dtype, int Ci, int Cx,
                       int x_off, int B, int D, int H, int W, int ksize, long long kchunk, float *part, float *g,
                       int accumulate, void *stream) {
  if (!dy || !x || !part || !g || kchunk < 1 || dy_off < 0 || dy_off + Co > Cdy || x_off < 0 || x_off + Ci > Cx)
    return gt::set_error(GT_ERR_ARG, "gt_nn_conv3d_wgrad: bad argument");
  const long long nvox = (long long)B * D * H * W;
  if (B < 1 || D < 1 || H < 1 || W < 1 || Co < 1 || Ci < 1)
    return gt::set_error(GT_ERR_ARG, "gt_nn_conv3d_wgrad: empty batch, volume or channel range");
  const long long nchunk = (nvox + kchunk - 1) / kchunk;
  if (nchunk > 65535) return gt::set_error(GT_ERR_ARG, "gt_nn_conv3d_wgrad: kchunk too small (more than 65535 chunks)");
  if ((ksize != 1 && ksize != 3) || (x_dtype != 0 && x_dtype != 1))
    return gt::set_error(GT_ERR_ARG, "gt_nn_conv3d_wgrad: ksize 1 or 3, dtype 0 or 1");
  const Shape s{B, D, H, W};
  cudaStream_t st = (cudaStream_t)stream;
  int nslot = 0;
  if (x_dtype == 1)
    NN_CK(wgrad<__nv_bfloat16>(ksize, dy, Co, Cdy, dy_off, x, Ci, Cx, x_off, s, nchunk, part, &nslot, st),
          "gt_nn_conv3d_wgrad");
  else
    NN_CK(wgrad<float>(ksize, dy, Co, Cdy, dy_off, x, Ci, Cx, x_off, s, nchunk, part, &nslot, st),
          "gt_nn_conv3d_wgrad");
  const long long n = (long long)Co * Ci * ksize * ksize * ksize;
  k_wgrad_reduce<<<nblk(n, 32), 256, 0, st>>>(part, nslot, n, g, accumulate);
  NN_CK(cudaGetLastError(), "gt_nn_conv3d_wgrad");
  return GT_OK;
}

int gt_nn_bias_grad(const float *dy, int Co, int Cdy, int dy_off, int B, long long vol, float *db, int accumulate,
                    void *stream) {
  if (!dy || !db || Co < 1 || dy_off < 0 || dy_off + Co > Cdy) return gt::set_error(GT_ERR_ARG, "gt_nn_bias_grad: bad argument");
  const int vec = vol % 4 == 0 && reinterpret_cast<size_t>(dy) % 16 == 0;
  if (B * vol <= BG_ONE)
    k_bias_grad<1><<<Co, 256, 0, (cudaStream_t)stream>>>(dy, Cdy, dy_off, vol, B, vec, db, accumulate);
  else
    k_bias_grad<BG_CL><<<(unsigned)Co * BG_CL, 256, 0, (cudaStream_t)stream>>>(dy, Cdy, dy_off, vol, B, vec, db, accumulate);
  NN_CK(cudaGetLastError(), "gt_nn_bias_grad");
  return GT_OK;
}

}  // extern "C"
