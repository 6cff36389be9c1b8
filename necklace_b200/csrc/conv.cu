// Convolution support kernels for channels-last (NHWC) bf16 activations, batch
// normalisation (training mode) fused with ReLU and the residual add, and pooling.
//
// A convolution is a GEMM on the tcgen05 kernel of gemm_sm100.cu:
//   1x1 stride 1      activations [N*H*W, Cin] are the A operand as they are;
//   C, Cout % 8 == 0  conv_sm100.cu reads the image itself where nkb_conv_route finds that quicker;
//   everything else   `im2col` gathers the receptive fields into col [N*Ho*Wo, KH*KW*Cin]
//                     (K index = (kh*KW + kw)*Cin + c, zero for padding), the weight is stored
//                     [Cout, KH*KW*Cin]; the data gradient is GEMM + `col2im` (written as a
//                     gather over the taps that touch an input pixel: no atomics, deterministic),
//                     the weight gradient is a GEMM over a recomputed col.
// The reference trains CNNs through torch's cuDNN convolutions
// (examples/dp/mnist/pytorch/main.py); these kernels take their place for the ResNet-50
// configuration.
#include <mutex>

#include "ptx.cuh"
#include "nkb_api.h"

namespace nkb {

static int conv_grid(long long work, int threads) {
  long long b = (work + threads - 1) / threads;
  const long long cap = 148LL * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

struct ConvGeom {
  int N, H, W, C, KH, KW, stride, pad, Ho, Wo, Kpad;
};

// VEC = 8: C % 8 == 0, 16-byte accesses; VEC = 1: any C.
template <int VEC>
__global__ void __launch_bounds__(256)
im2col_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ col, ConvGeom g) {
  if (!grid_dep_begin()) return;
  const long long M = (long long)g.N * g.Ho * g.Wo;
  const int kchunks = g.Kpad / VEC;
  const int Kreal = g.KH * g.KW * g.C;
  const long long total = M * kchunks;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += stride) {
    const long long m = idx / kchunks;
    const int k = (int)(idx % kchunks) * VEC;
    const int wo = (int)(m % g.Wo);
    const long long t = m / g.Wo;
    const int ho = (int)(t % g.Ho);
    const int n = (int)(t / g.Ho);
    bool ok = k < Kreal;
    long long src = 0;
    if (ok) {
      const int tap = k / g.C, c = k % g.C;
      const int kh = tap / g.KW, kw = tap % g.KW;
      const int h = ho * g.stride - g.pad + kh, w = wo * g.stride - g.pad + kw;
      ok = h >= 0 && h < g.H && w >= 0 && w < g.W;
      src = (((long long)n * g.H + h) * g.W + w) * g.C + c;
    }
    const long long x_elems = (long long)g.N * g.H * g.W * g.C;
    if (ok && !NKB_IN_BOUNDS(src + VEC - 1, x_elems)) ok = false;
    if (!NKB_IN_BOUNDS(m * g.Kpad + k + VEC - 1, M * g.Kpad)) continue;
    if (VEC == 8) {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (ok) v = *reinterpret_cast<const uint4*>(x + src);
      *reinterpret_cast<uint4*>(col + m * g.Kpad + k) = v;
    } else {
      col[m * g.Kpad + k] = ok ? x[src] : __float2bfloat16(0.f);
    }
  }
}

// Channel counts that are not a multiple of 8 (the 3-channel stem).  A block gathers `tw`
// neighbouring output pixels of one row: the KH input rows that they share come into shared
// memory once (with the padding as zeros), a table says where each of a pixel's Kpad entries
// lies there, and a thread puts eight of them together for one 16-byte store.  (Gathering
// from global memory, 2 bytes and two divisions per entry, took 1375 us for the 224 x 224 stem
// of 256 images; now 484 us, the 976 MB that it writes take 150 us.)
constexpr int IM2COL_TILE_SMEM = 40 * 1024;
__global__ void __launch_bounds__(256)
im2col_tile_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ col, ConvGeom g,
                   int tw, int row_elems, int tiles_w) {
  if (!grid_dep_begin()) return;
  extern __shared__ __align__(16) uint16_t ic_smem[];
  uint16_t* table = ic_smem;                       // [Kpad]: offset of entry k, pixel 0
  uint16_t* rows = ic_smem + g.Kpad;               // [KH][row_elems], then 8 zeros
  const int wo0 = (blockIdx.x % tiles_w) * tw;
  const int ho = (blockIdx.x / tiles_w) % g.Ho;
  const int n = blockIdx.x / tiles_w / g.Ho;
  const int kc = g.KW * g.C, Kreal = g.KH * kc;
  const int zero = g.KH * row_elems;
  for (int k = threadIdx.x; k < g.Kpad; k += 256)
    table[k] = (uint16_t)(k < Kreal ? (k / kc) * row_elems + k % kc : zero);
  const int e0 = (wo0 * g.stride - g.pad) * g.C;   // element of the input row that lies at 0
  const int WC = g.W * g.C;
  for (int kh = 0; kh < g.KH; ++kh) {
    const int h = ho * g.stride - g.pad + kh;
    const bool in = h >= 0 && h < g.H;
    const uint16_t* src = reinterpret_cast<const uint16_t*>(x) +
                          ((long long)n * g.H + (in ? h : 0)) * WC;
    for (int e = threadIdx.x; e < row_elems; e += 256) {
      const int w = e0 + e;
      const bool ok = in && w >= 0 && w < WC &&
                      NKB_IN_BOUNDS(((long long)n * g.H + h) * WC + w, (long long)g.N * g.H * WC);
      rows[kh * row_elems + e] = ok ? src[w] : (uint16_t)0;
    }
  }
  if (threadIdx.x == 0) rows[zero] = 0;
  __syncthreads();
  const int px = min(tw, g.Wo - wo0), chunks = g.Kpad >> 3, sc = g.stride * g.C;
  const long long out0 = (((long long)n * g.Ho + ho) * g.Wo + wo0) * chunks;
  uint4* out = reinterpret_cast<uint4*>(col) + out0;
  for (int i = threadIdx.x; i < px * chunks; i += 256) {
    const int p = i / chunks, k = (i - p * chunks) * 8;
    const uint4 t = *reinterpret_cast<const uint4*>(table + k);
    const uint32_t tt[4] = {t.x, t.y, t.z, t.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = tt[j] & 0xffff, b = tt[j] >> 16;
      const uint32_t lo = rows[a == zero ? zero : a + p * sc];
      const uint32_t hi = rows[b == zero ? zero : b + p * sc];
      o[j] = lo | hi << 16;
    }
    if (NKB_IN_BOUNDS(out0 + i, (long long)g.N * g.Ho * g.Wo * chunks))
      out[i] = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

// dx[n,h,w,c] = sum over taps (kh,kw) with (h + pad - kh) % stride == 0 (same for w) of
// dcol[(n, (h+pad-kh)/stride, (w+pad-kw)/stride), (kh*KW+kw)*C + c]
template <int VEC>
__global__ void __launch_bounds__(256)
col2im_kernel(const __nv_bfloat16* __restrict__ dcol, __nv_bfloat16* __restrict__ dx, ConvGeom g) {
  if (!grid_dep_begin()) return;
  const int cchunks = g.C / VEC;
  const long long total = (long long)g.N * g.H * g.W * cchunks;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += stride) {
    const int c = (int)(idx % cchunks) * VEC;
    long long t = idx / cchunks;
    const int w = (int)(t % g.W);
    t /= g.W;
    const int h = (int)(t % g.H);
    const int n = (int)(t / g.H);
    float acc[VEC];
#pragma unroll
    for (int j = 0; j < VEC; ++j) acc[j] = 0.f;
    for (int kh = 0; kh < g.KH; ++kh) {
      const int hn = h + g.pad - kh;
      if (hn < 0 || hn % g.stride) continue;
      const int ho = hn / g.stride;
      if (ho >= g.Ho) continue;
      for (int kw = 0; kw < g.KW; ++kw) {
        const int wn = w + g.pad - kw;
        if (wn < 0 || wn % g.stride) continue;
        const int wo = wn / g.stride;
        if (wo >= g.Wo) continue;
        const long long src = (((long long)n * g.Ho + ho) * g.Wo + wo) * g.Kpad +
                              (long long)(kh * g.KW + kw) * g.C + c;
        if (!NKB_IN_BOUNDS(src + VEC - 1, (long long)g.N * g.Ho * g.Wo * g.Kpad)) continue;
        if (VEC == 8) {
          uint4 v = *reinterpret_cast<const uint4*>(dcol + src);
          uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 f = unpack_bf16x2(u[j]);
            acc[2 * j] += f.x;
            acc[2 * j + 1] += f.y;
          }
        } else {
          acc[0] += __bfloat162float(dcol[src]);
        }
      }
    }
    const long long dst = (((long long)n * g.H + h) * g.W + w) * g.C + c;
    if (VEC == 8) {
      *reinterpret_cast<uint4*>(dx + dst) =
          make_uint4(pack_bf16x2(acc[0], acc[1]), pack_bf16x2(acc[2], acc[3]),
                     pack_bf16x2(acc[4], acc[5]), pack_bf16x2(acc[6], acc[7]));
    } else {
      dx[dst] = __float2bfloat16(acc[0]);
    }
  }
}

// ------------------------------------------------------------------ batch norm
// Per-channel sums over the rows of a [M, C] matrix (C % 8 == 0):
//   MODE 0: acc[0][c] += sum x,        acc[1][c] += sum x^2            (forward statistics)
//   MODE 1: acc[0][c] += sum dy',      acc[1][c] += sum dy' * xhat     (backward sums)
// with dy' = dy * (y > 0) when relu, xhat = (x - mean) * rstd.  The signs of the layer's output
// are kept as one bit per element (`mask`, one byte per thread and row): the backward kernels
// are bound by memory and the output itself would be a third of what they read.
// Threads: 8 channels each; a block covers `cx` channel chunks x `ry` row lanes.
//
// Each thread loads BN_ROWS rows before it uses the first: with one row in flight the 1024
// threads of an SM (64 registers) kept 32 KB on the way, less than the latency of the
// memory times its rate.
//
// With one operation per value these kernels took half or more of an SM's issue slots (apply 62 %), so
// values travel as packed fp32 pairs and the masks are made and applied on words of two bf16.  256
// images of 56 x 56 x 256: apply 148 -> 131 us, backward sums 139 -> 134, backward apply 198 -> 191;
// evaluation 145 -> 132 us.
constexpr int BN_ROWS = 4;

// Bits 2 j and 2 j + 1 of a byte of signs as a mask of the two halves of word j.
struct BnMask {
  uint32_t lo, hi;  // bits 0-3 and 4-7 of the byte as the top bits of four bytes
  // (the products of the four bits with the four shifts fall on different bits)
  __device__ __forceinline__ explicit BnMask(uint32_t m)
      : lo((m & 15u) * 0x10204080u), hi((m >> 4) * 0x10204080u) {}
  __device__ __forceinline__ uint32_t word(int j) const {  // j is a constant of the caller
    uint32_t r;  // bit 3 of a selector spreads the byte's top bit over the byte
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(j < 2 ? lo : hi), "r"(j & 1 ? 0xBBAA : 0x9988));
    return r;
  }
};

template <int MODE>
__global__ void __launch_bounds__(256)
bn_sums_kernel(const __nv_bfloat16* __restrict__ a, const __nv_bfloat16* __restrict__ x,
               const uint8_t* __restrict__ mask, const float* __restrict__ stats,
               float* __restrict__ acc, long long M, int C, int cx) {
  if (!grid_dep_begin()) return;
  __shared__ float sh[2][256][8 + 1];
  const int ry = 256 / cx;
  const int tx = threadIdx.x % cx, ty = threadIdx.x / cx;
  const int c = (blockIdx.x * cx + tx) * 8;
  float s0[8], s1[8];
  f32x2_t t0[4], t1[4];  // MODE 1 (the forward sums gain nothing from pairs: 79 us, packed 83)
#pragma unroll
  for (int j = 0; j < 8; ++j) s0[j] = s1[j] = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) t0[j] = t1[j] = f2_pack(0.f, 0.f);
  if (c < C && ty < ry) {
    f32x2_t neg_mean[4];
    if (MODE == 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) neg_mean[j] = f2_pack(-stats[c + 2 * j], -stats[c + 2 * j + 1]);
    }
    const long long step = (long long)gridDim.y * ry;
    for (long long q = (long long)blockIdx.y * ry + ty; q < M; q += BN_ROWS * step) {
      uint4 va[BN_ROWS], vx[BN_ROWS];
      uint32_t m[BN_ROWS];
#pragma unroll
      for (int u = 0; u < BN_ROWS; ++u) {
        // the backward sums go from the last row, which the kernel before has just written, to the
        // first, with which the one behind begins: either finds a part of the rows in L2
        const long long row = MODE == 1 ? M - 1 - (q + u * step) : q + u * step;
        const long long off = row * C + c;
        va[u] = vx[u] = make_uint4(0, 0, 0, 0);
        m[u] = 0xffu;
        if (q + u * step < M) {
          va[u] = *reinterpret_cast<const uint4*>(a + off);
          if (MODE == 1) {
            vx[u] = *reinterpret_cast<const uint4*>(x + off);
            if (mask) m[u] = mask[off >> 3];
          }
        }
      }
#pragma unroll
      for (int u = 0; u < BN_ROWS; ++u) {
        const uint32_t ua[4] = {va[u].x, va[u].y, va[u].z, va[u].w};
        const uint32_t ux[4] = {vx[u].x, vx[u].y, vx[u].z, vx[u].w};
        const BnMask keep(m[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (MODE == 0) {
            const float2 f = unpack_bf16x2(ua[j]);
            s0[2 * j] += f.x;
            s0[2 * j + 1] += f.y;
            s1[2 * j] += f.x * f.x;
            s1[2 * j + 1] += f.y * f.y;
          } else {
            // rows outside have f = 0
            const f32x2_t f = f2_from_bf16x2(ua[j] & keep.word(j));
            t0[j] = f2_add(t0[j], f);
            t1[j] = f2_fma(f, f2_add(f2_from_bf16x2(ux[j]), neg_mean[j]), t1[j]);
          }
        }
      }
    }
    if (MODE == 1) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f2_unpack(t0[j], s0[2 * j], s0[2 * j + 1]);
        f2_unpack(t1[j], s1[2 * j], s1[2 * j + 1]);
        s1[2 * j] *= stats[C + c + 2 * j];
        s1[2 * j + 1] *= stats[C + c + 2 * j + 1];
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) { sh[0][threadIdx.x][j] = s0[j]; sh[1][threadIdx.x][j] = s1[j]; }
  __syncthreads();
  // the first cx*8 threads each own one channel of the strip and add up the row lanes
  if (threadIdx.x < cx * 8) {
    const int chunk = threadIdx.x / 8, j = threadIdx.x % 8;
    const int cc = (blockIdx.x * cx + chunk) * 8 + j;
    if (cc < C) {
      float t0 = 0.f, t1 = 0.f;
      for (int l = 0; l < ry; ++l) {
        t0 += sh[0][l * cx + chunk][j];
        t1 += sh[1][l * cx + chunk][j];
      }
      atomicAdd(acc + cc, t0);
      atomicAdd(acc + C + cc, t1);
    }
  }
}

// stats[0][c] = mean, stats[1][c] = rstd from the forward sums; running statistics updated
// (momentum form of torch.nn.BatchNorm2d, unbiased variance); the accumulator is re-zeroed.
__global__ void bn_finalize_kernel(float* __restrict__ acc, float* __restrict__ stats,
                                   float* __restrict__ run_mean, float* __restrict__ run_var,
                                   long long M, int C, float eps, float momentum) {
  if (!grid_dep_begin()) return;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const float inv = 1.f / (float)M;
  const float mean = acc[c] * inv;
  float var = acc[C + c] * inv - mean * mean;
  var = fmaxf(var, 0.f);
  stats[c] = mean;
  stats[C + c] = rsqrtf(var + eps);
  if (run_mean) {
    const float unb = M > 1 ? var * (float)M / (float)(M - 1) : var;
    run_mean[c] = (1.f - momentum) * run_mean[c] + momentum * mean;
    run_var[c] = (1.f - momentum) * run_var[c] + momentum * unb;
  }
  acc[c] = 0.f;
  acc[C + c] = 0.f;
}

// y = act((x - mean) * rstd * gamma + beta (+ res)).  Thread layout as in bn_sums_kernel: a
// thread owns 8 fixed channels (its per-channel constants stay in registers) and walks rows.
__global__ void __launch_bounds__(256)
bn_apply_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ mean,
                const float* __restrict__ spread, float eps,
                const __nv_bfloat16* __restrict__ gamma, const __nv_bfloat16* __restrict__ beta,
                const __nv_bfloat16* __restrict__ res, __nv_bfloat16* __restrict__ y,
                uint8_t* __restrict__ mask, long long M, int C, int cx, int relu) {
  if (!grid_dep_begin()) return;
  const int ry = 256 / cx;
  const int tx = threadIdx.x % cx, ty = threadIdx.x / cx;
  const int c = (blockIdx.x * cx + tx) * 8;
  if (c >= C || ty >= ry) return;
  f32x2_t sc2[4], sh2[4];
  {
    uint4 vg = *reinterpret_cast<const uint4*>(gamma + c);
    uint4 vb = *reinterpret_cast<const uint4*>(beta + c);
    uint32_t ug[4] = {vg.x, vg.y, vg.z, vg.w}, ub[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 fg = unpack_bf16x2(ug[j]), fb = unpack_bf16x2(ub[j]);
      // spread: rstd, or the variance when eps >= 0; rsqrtf gives the bits of torch.rsqrt, so both
      // ways of evaluating a layer agree (a correctly rounded root moved bf16 roundings that
      // fifty layers carried to 0.3 % of ResNet-50's logits)
      const float r0 = spread[c + 2 * j], r1 = spread[c + 2 * j + 1];
      const float a = (eps < 0.f ? r0 : rsqrtf(r0 + eps)) * fg.x;
      const float b = (eps < 0.f ? r1 : rsqrtf(r1 + eps)) * fg.y;
      sc2[j] = f2_pack(a, b);
      sh2[j] = f2_pack(fb.x - mean[c + 2 * j] * a, fb.y - mean[c + 2 * j + 1] * b);
    }
  }
  const long long step = (long long)gridDim.y * ry;
  for (long long r = (long long)blockIdx.y * ry + ty; r < M; r += BN_ROWS * step) {
    uint4 vx[BN_ROWS], vr[BN_ROWS];
#pragma unroll
    for (int u = 0; u < BN_ROWS; ++u) {
      const long long off = (r + u * step) * C + c;
      vr[u] = make_uint4(0, 0, 0, 0);
      if (r + u * step < M) {
        vx[u] = *reinterpret_cast<const uint4*>(x + off);
        if (res) vr[u] = *reinterpret_cast<const uint4*>(res + off);
      }
    }
#pragma unroll
    for (int u = 0; u < BN_ROWS; ++u) {
      if (r + u * step >= M) break;
      const long long off = (r + u * step) * C + c;
      const uint32_t ux[4] = {vx[u].x, vx[u].y, vx[u].z, vx[u].w};
      const uint32_t ur[4] = {vr[u].x, vr[u].y, vr[u].z, vr[u].w};
      uint32_t o[4];
      uint32_t m = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        f32x2_t v = f2_fma(f2_from_bf16x2(ux[j]), sc2[j], sh2[j]);
        if (res) v = f2_add(v, f2_from_bf16x2(ur[j]));
        o[j] = f2_to_bf16x2(v);
        // the larger of the rounded value and 0 is the rounded value of the larger
        uint32_t pos;
        asm("max.bf16x2 %0, %1, %2;" : "=r"(pos) : "r"(o[j]), "r"(0));
        if (relu) o[j] = pos;
        // What a comparison of the stored value with zero gives: a half is 0 or 1 .. 0x7f80 now, and
        // adding 0x7fff sets its top bit unless it is 0.  Bits 2 j and 2 j + 16.
        m |= ((pos + 0x7fff7fffu) >> (15 - 2 * j)) & (0x00010001u << (2 * j));
      }
      *reinterpret_cast<uint4*>(y + off) = make_uint4(o[0], o[1], o[2], o[3]);
      if (mask) mask[off >> 3] = (uint8_t)(m | m >> 15);
    }
  }
}

// dx = gamma * rstd * (dy' - s0/M - xhat * s1/M);  dres = dy' (optional);
// sums = [2][C] from bn_sums_kernel<1>.  Same thread layout.
__global__ void __launch_bounds__(256)
bn_bwd_apply_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                    const uint8_t* __restrict__ mask, const float* __restrict__ stats,
                    const float* __restrict__ sums, const __nv_bfloat16* __restrict__ gamma,
                    __nv_bfloat16* __restrict__ dx, __nv_bfloat16* __restrict__ dres, long long M,
                    int C, int cx) {
  if (!grid_dep_begin()) return;
  const int ry = 256 / cx;
  const int tx = threadIdx.x % cx, ty = threadIdx.x / cx;
  const int c = (blockIdx.x * cx + tx) * 8;
  if (c >= C || ty >= ry) return;
  const float invM = 1.f / (float)M;
  // dx = k1 * dy' + k2 * x + k3 with k1 = gamma rstd, k2 = -k1 rstd s1/M,
  // k3 = -k1 (s0/M - mean rstd s1/M)
  f32x2_t k1[4], k2[4], k3[4];
  {
    uint4 vg = *reinterpret_cast<const uint4*>(gamma + c);
    uint32_t ug[4] = {vg.x, vg.y, vg.z, vg.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 fg = unpack_bf16x2(ug[j]);
      float q1[2], q2[2], q3[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int ch = c + 2 * j + e;
        const float mean = stats[ch], rstd = stats[C + ch];
        const float a0 = sums[ch] * invM, a1 = sums[C + ch] * invM;
        q1[e] = (e ? fg.y : fg.x) * rstd;
        q2[e] = -q1[e] * rstd * a1;
        q3[e] = -q1[e] * (a0 - mean * rstd * a1);
      }
      k1[j] = f2_pack(q1[0], q1[1]);
      k2[j] = f2_pack(q2[0], q2[1]);
      k3[j] = f2_pack(q3[0], q3[1]);
    }
  }
  constexpr int U = BN_ROWS / 2;
  const long long step = (long long)gridDim.y * ry;
  for (long long r = (long long)blockIdx.y * ry + ty; r < M; r += U * step) {
    uint4 vd[U], vx[U];
    uint32_t mk[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long off = (r + u * step) * C + c;
      if (r + u * step < M) {
        vd[u] = *reinterpret_cast<const uint4*>(dy + off);
        vx[u] = *reinterpret_cast<const uint4*>(x + off);
        mk[u] = mask ? mask[off >> 3] : 0xffu;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (r + u * step >= M) break;
      const long long off = (r + u * step) * C + c;
      const uint32_t ud[4] = {vd[u].x, vd[u].y, vd[u].z, vd[u].w};
      const uint32_t ux[4] = {vx[u].x, vx[u].y, vx[u].z, vx[u].w};
      const BnMask keep(mk[u]);
      uint32_t o[4], rr[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        rr[j] = ud[j] & keep.word(j);
        o[j] = f2_to_bf16x2(f2_fma(k1[j], f2_from_bf16x2(rr[j]),
                                   f2_fma(k2[j], f2_from_bf16x2(ux[j]), k3[j])));
      }
      *reinterpret_cast<uint4*>(dx + off) = make_uint4(o[0], o[1], o[2], o[3]);
      if (dres) *reinterpret_cast<uint4*>(dres + off) = make_uint4(rr[0], rr[1], rr[2], rr[3]);
    }
  }
}

// dgamma / dbeta (bf16, written or accumulated) from the backward sums; sums re-zeroed.
__global__ void bn_param_grad_kernel(float* __restrict__ sums, __nv_bfloat16* __restrict__ dgamma,
                                     __nv_bfloat16* __restrict__ dbeta, int C, int acc_g,
                                     int acc_b) {
  if (!grid_dep_begin()) return;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  float g = sums[C + c], b = sums[c];
  if (dgamma) {
    if (acc_g) g += __bfloat162float(dgamma[c]);
    dgamma[c] = __float2bfloat16(g);
  }
  if (dbeta) {
    if (acc_b) b += __bfloat162float(dbeta[c]);
    dbeta[c] = __float2bfloat16(b);
  }
  sums[c] = 0.f;
  sums[C + c] = 0.f;
}

// --------------------------------------------------------------------- pooling
// 3x3 / stride 2 / pad 1 max pooling, NHWC, C % 8 == 0; idx = winning tap (0..8) per element.
__global__ void __launch_bounds__(256)
maxpool_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y,
                   uint8_t* __restrict__ idx, int N, int H, int W, int C, int Ho, int Wo) {
  if (!grid_dep_begin()) return;
  const int cch = C / 8;
  const long long total = (long long)N * Ho * Wo * cch;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
    const int c = (int)(i % cch) * 8;
    long long t = i / cch;
    const int wo = (int)(t % Wo);
    t /= Wo;
    const int ho = (int)(t % Ho);
    const int n = (int)(t / Ho);
    float best[8];
    int arg[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) { best[j] = -INFINITY; arg[j] = 0; }
    for (int kh = 0; kh < 3; ++kh) {
      const int h = ho * 2 - 1 + kh;
      if (h < 0 || h >= H) continue;
      for (int kw = 0; kw < 3; ++kw) {
        const int w = wo * 2 - 1 + kw;
        if (w < 0 || w >= W) continue;
        const long long src = (((long long)n * H + h) * W + w) * C + c;
        if (!NKB_IN_BOUNDS(src + 7, (long long)N * H * W * C)) continue;
        uint4 v = *reinterpret_cast<const uint4*>(x + src);
        uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float2 f = unpack_bf16x2(u[j]);
          if (f.x > best[2 * j]) { best[2 * j] = f.x; arg[2 * j] = kh * 3 + kw; }
          if (f.y > best[2 * j + 1]) { best[2 * j + 1] = f.y; arg[2 * j + 1] = kh * 3 + kw; }
        }
      }
    }
    const long long dst = (((long long)n * Ho + ho) * Wo + wo) * C + c;
    *reinterpret_cast<uint4*>(y + dst) =
        make_uint4(pack_bf16x2(best[0], best[1]), pack_bf16x2(best[2], best[3]),
                   pack_bf16x2(best[4], best[5]), pack_bf16x2(best[6], best[7]));
    uint32_t lo = arg[0] | (arg[1] << 8) | (arg[2] << 16) | (arg[3] << 24);
    uint32_t hi = arg[4] | (arg[5] << 8) | (arg[6] << 16) | (arg[7] << 24);
    *reinterpret_cast<uint2*>(idx + dst) = make_uint2(lo, hi);
  }
}

// A thread makes the 2 x 2 input positions (2i.., 2j..) of 8 channels from the four windows that
// touch them: each window is loaded for 4 positions instead of being looked for by each of the
// up to 9 it covers (411 MB of dx for 256 images took 407 us, now 220 us; the traffic takes
// 86 us).
__global__ void __launch_bounds__(256)
maxpool_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const uint8_t* __restrict__ idx,
                   __nv_bfloat16* __restrict__ dx, int N, int H, int W, int C, int Ho, int Wo) {
  if (!grid_dep_begin()) return;
  const int cch = C / 8, Hb = (H + 1) / 2, Wb = (W + 1) / 2;
  const long long total = (long long)N * Hb * Wb * cch;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < total; q += stride) {
    const int c = (int)(q % cch) * 8;
    long long t = q / cch;
    const int j = (int)(t % Wb);
    t /= Wb;
    const int i = (int)(t % Hb);
    const int n = (int)(t / Hb);
    uint4 v[4];
    uint2 iv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {  // window (i + k / 2, j + k % 2)
      const int ho = i + (k >> 1), wo = j + (k & 1);
      v[k] = make_uint4(0, 0, 0, 0);
      iv[k] = make_uint2(~0u, ~0u);  // no tap
      if (ho < Ho && wo < Wo) {
        const long long src = (((long long)n * Ho + ho) * Wo + wo) * C + c;
        if (!NKB_IN_BOUNDS(src + 7, (long long)N * Ho * Wo * C)) continue;
        v[k] = *reinterpret_cast<const uint4*>(dy + src);
        iv[k] = *reinterpret_cast<const uint2*>(idx + src);
      }
    }
    float acc[4][8];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[p][e] = 0.f;
#pragma unroll
    for (int k = 3; k >= 0; --k) {  // (taps in ascending order for every position)
      const uint32_t u[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float2 f = unpack_bf16x2(u[e >> 1]);
        const float val = (e & 1) ? f.y : f.x;
        const uint32_t tap = ((e < 4 ? iv[k].x : iv[k].y) >> (8 * (e & 3))) & 0xff;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          // row 0 is tap 1 of window row i; row 1 is tap 2 of it and tap 0 of row i + 1
          const int dh = k >> 1, dw = k & 1, r = p >> 1, s = p & 1;
          if (r + 1 - 2 * dh < 0 || s + 1 - 2 * dw < 0) continue;
          if (tap == (uint32_t)((r + 1 - 2 * dh) * 3 + s + 1 - 2 * dw)) acc[p][e] += val;
        }
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int h = 2 * i + (p >> 1), w = 2 * j + (p & 1);
      if (h < H && w < W)
        *reinterpret_cast<uint4*>(dx + (((long long)n * H + h) * W + w) * C + c) =
            make_uint4(pack_bf16x2(acc[p][0], acc[p][1]), pack_bf16x2(acc[p][2], acc[p][3]),
                       pack_bf16x2(acc[p][4], acc[p][5]), pack_bf16x2(acc[p][6], acc[p][7]));
    }
  }
}

// Global average pooling over HW: x [N, HW, C] -> y [N, C]; backward spreads dy / HW.
__global__ void __launch_bounds__(256)
avgpool_fwd_kernel(const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ y, int N,
                   int HW, int C) {
  if (!grid_dep_begin()) return;
  const int cch = C / 8;
  const long long total = (long long)N * cch;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % cch) * 8;
    const int n = (int)(i / cch);
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int p = 0; p < HW; ++p) {
      uint4 v = *reinterpret_cast<const uint4*>(x + ((long long)n * HW + p) * C + c);
      uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 f = unpack_bf16x2(u[j]);
        acc[2 * j] += f.x;
        acc[2 * j + 1] += f.y;
      }
    }
    const float inv = 1.f / (float)HW;
    *reinterpret_cast<uint4*>(y + (long long)n * C + c) =
        make_uint4(pack_bf16x2(acc[0] * inv, acc[1] * inv), pack_bf16x2(acc[2] * inv, acc[3] * inv),
                   pack_bf16x2(acc[4] * inv, acc[5] * inv), pack_bf16x2(acc[6] * inv, acc[7] * inv));
  }
}

__global__ void __launch_bounds__(256)
avgpool_bwd_kernel(const __nv_bfloat16* __restrict__ dy, __nv_bfloat16* __restrict__ dx, int N,
                   int HW, int C) {
  if (!grid_dep_begin()) return;
  const int cch = C / 8;
  const long long total = (long long)N * HW * cch;
  const float inv = 1.f / (float)HW;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % cch) * 8;
    const long long t = i / cch;
    const int n = (int)(t / HW);
    uint4 v = *reinterpret_cast<const uint4*>(dy + (long long)n * C + c);
    uint32_t u[4] = {v.x, v.y, v.z, v.w}, o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = unpack_bf16x2(u[j]);
      o[j] = pack_bf16x2(f.x * inv, f.y * inv);
    }
    *reinterpret_cast<uint4*>(dx + t * C + c) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

}  // namespace nkb

using namespace nkb;

static ConvGeom geom(int N, int H, int W, int C, int KH, int KW, int stride, int pad, int Kpad) {
  ConvGeom g;
  g.N = N; g.H = H; g.W = W; g.C = C; g.KH = KH; g.KW = KW; g.stride = stride; g.pad = pad;
  g.Ho = (H + 2 * pad - KH) / stride + 1;
  g.Wo = (W + 2 * pad - KW) / stride + 1;
  g.Kpad = Kpad;
  return g;
}

// Output pixels per block of im2col_tile_kernel: at most 64, as many as shared memory (and the
// table's 16-bit offsets) hold; 0 where one pixel's window does not fit or the grid would be
// larger than a launch takes.
static int im2col_tile(const ConvGeom& g) {
  for (int tw = g.Wo < 64 ? g.Wo : 64; tw >= 1; tw >>= 1) {
    const long long elems = (long long)g.KH * (((tw - 1) * g.stride + g.KW) * (long long)g.C);
    if (2 * (g.Kpad + elems + 8) > IM2COL_TILE_SMEM || elems > 65000) continue;
    const long long blocks = (long long)((g.Wo + tw - 1) / tw) * g.Ho * g.N;
    return blocks < (1LL << 31) ? tw : 0;
  }
  return 0;
}

extern "C" int nkb_im2col_nhwc(const void* x, void* col, int N, int H, int W, int C, int KH,
                               int KW, int stride, int pad, int Kpad, void* stream) {
  if (Kpad < KH * KW * C || (Kpad & 7)) return -3;
  ConvGeom g = geom(N, H, W, C, KH, KW, stride, pad, Kpad);
  if (g.Ho <= 0 || g.Wo <= 0) return -2;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const long long M = (long long)N * g.Ho * g.Wo;
  const bool vec = (C % 8 == 0) && !(reinterpret_cast<uintptr_t>(x) & 15) &&
                   !(reinterpret_cast<uintptr_t>(col) & 15);
  if (vec) {
    launch_dep(im2col_kernel<8>, conv_grid(M * (Kpad / 8), 256), 256, 0, s,
               static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(col), g);
  } else if (int tw = im2col_tile(g); tw > 0 && !(reinterpret_cast<uintptr_t>(col) & 15)) {
    const int row_elems = ((tw - 1) * stride + KW) * C, tiles_w = (g.Wo + tw - 1) / tw;
    launch_dep(im2col_tile_kernel, (unsigned)(tiles_w * (long long)g.Ho * N), 256,
               2 * (Kpad + KH * row_elems + 8), s, static_cast<const __nv_bfloat16*>(x),
               static_cast<__nv_bfloat16*>(col), g, tw, row_elems, tiles_w);
  } else {
    launch_dep(im2col_kernel<1>, conv_grid(M * Kpad, 256), 256, 0, s,
               static_cast<const __nv_bfloat16*>(x), static_cast<__nv_bfloat16*>(col), g);
  }
  return (int)cudaGetLastError();
}

extern "C" int nkb_col2im_nhwc(const void* dcol, void* dx, int N, int H, int W, int C, int KH,
                               int KW, int stride, int pad, int Kpad, void* stream) {
  if (Kpad < KH * KW * C || (Kpad & 7)) return -3;
  ConvGeom g = geom(N, H, W, C, KH, KW, stride, pad, Kpad);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool vec = (C % 8 == 0) && !(reinterpret_cast<uintptr_t>(dx) & 15) &&
                   !(reinterpret_cast<uintptr_t>(dcol) & 15);
  const long long px = (long long)N * H * W;
  if (vec)
    launch_dep(col2im_kernel<8>, conv_grid(px * (C / 8), 256), 256, 0, s,
               static_cast<const __nv_bfloat16*>(dcol), static_cast<__nv_bfloat16*>(dx), g);
  else
    launch_dep(col2im_kernel<1>, conv_grid(px * C, 256), 256, 0, s,
               static_cast<const __nv_bfloat16*>(dcol), static_cast<__nv_bfloat16*>(dx), g);
  return (int)cudaGetLastError();
}

static void bn_sums_dims(long long M, int C, int& cx, dim3& grid) {
  // strips of at most 32 chunks of 8 channels, all of the same width: with widths in powers of two
  // the 17 chunks of 136 channels were a strip of 16 and one of a single chunk, whose blocks held
  // their place on the SM with one lane in 16 (802816 rows: evaluation 138 -> 81 us, there and back
  // 456 -> 313 us).  The threads behind cx * ry (at most cx - 1) have no row.
  const int chunks = C / 8;
  const int gx = (chunks + 31) / 32;
  cx = (chunks + gx - 1) / gx;
  const int ry = 256 / cx;
  // six blocks per SM: one round of the forward sums (40 registers), two of the others (80)
  long long gy = (148LL * 6) / gx;
  const long long need = (M + ry - 1) / ry;
  if (gy > need) gy = need;
  if (gy < 1) gy = 1;
  if (gy > 65535) gy = 65535;
  grid = dim3(gx, (unsigned)gy);
}

// Forward: batch statistics of x [M, C], then y = act(bn(x) (+ res)).  acc: fp32 [2][C], zero on
// entry, left zero.  stats out: fp32 [2][C] (mean, rstd).  mask (optional): one bit per element,
// y > 0, in [M * C / 8] bytes, bit j of byte i for element 8 i + j.
//
// The kernels of a call hand their sums on through `acc`, which calls on one stream share: no other
// thread's call on that stream may come between them.
static std::mutex g_bn_order;
extern "C" int nkb_bn_fwd(const void* x, const void* gamma, const void* beta, const void* res,
                          void* y, void* mask, float* stats, float* acc, float* run_mean,
                          float* run_var, long long M, int C, float eps, float momentum, int relu,
                          void* stream) {
  if (C % 8) return -3;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y) |
       reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta)) & 15)
    return -3;
  if (res && (reinterpret_cast<uintptr_t>(res) & 15)) return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int cx;
  dim3 grid;
  bn_sums_dims(M, C, cx, grid);
  std::lock_guard<std::mutex> order(g_bn_order);
  launch_dep(bn_sums_kernel<0>, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(x), nullptr,
             nullptr, nullptr, acc, M, C, cx);
  launch_dep(bn_finalize_kernel, (C + 127) / 128, 128, 0, s, acc, stats, run_mean, run_var, M, C,
             eps, momentum);
  launch_dep(bn_apply_kernel, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(x), stats,
             stats + C, -1.f, static_cast<const __nv_bfloat16*>(gamma),
             static_cast<const __nv_bfloat16*>(beta), static_cast<const __nv_bfloat16*>(res),
             static_cast<__nv_bfloat16*>(y), static_cast<uint8_t*>(mask), M, C, cx, relu);
  return (int)cudaGetLastError();
}

// Evaluation mode: y = act((x - mean) * rstd * gamma + beta (+ res)) with given stats [2][C].
extern "C" int nkb_bn_apply(const void* x, const float* stats, const void* gamma, const void* beta,
                            const void* res, void* y, long long M, int C, int relu, void* stream) {
  if (C % 8) return -3;
  int cx;
  dim3 grid;
  bn_sums_dims(M, C, cx, grid);
  launch_dep(bn_apply_kernel, grid, 256, 0, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(x), stats, stats + C, -1.f,
             static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta),
             static_cast<const __nv_bfloat16*>(res), static_cast<__nv_bfloat16*>(y), nullptr, M, C,
             cx, relu);
  return (int)cudaGetLastError();
}

// The same from running statistics: rstd is taken in the kernel (three single-operation kernels
// per layer made (mean, rstd) of them before).
extern "C" int nkb_bn_eval(const void* x, const float* run_mean, const float* run_var, float eps,
                           const void* gamma, const void* beta, const void* res, void* y,
                           long long M, int C, int relu, void* stream) {
  if (C % 8 || eps < 0.f) return -3;
  int cx;
  dim3 grid;
  bn_sums_dims(M, C, cx, grid);
  launch_dep(bn_apply_kernel, grid, 256, 0, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(x), run_mean, run_var, eps,
             static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta),
             static_cast<const __nv_bfloat16*>(res), static_cast<__nv_bfloat16*>(y), nullptr, M, C,
             cx, relu);
  return (int)cudaGetLastError();
}

// Backward: dx (and dres = dy masked by the ReLU when given), dgamma / dbeta written or
// accumulated.  mask: what the forward wrote, null without a ReLU.
extern "C" int nkb_bn_bwd(const void* dy, const void* x, const void* mask, const float* stats,
                          const void* gamma, void* dx, void* dres, void* dgamma, void* dbeta,
                          int acc_g, int acc_b, float* acc, long long M, int C, void* stream) {
  if (C % 8) return -3;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(x) |
       reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(gamma)) & 15)
    return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int cx;
  dim3 grid;
  bn_sums_dims(M, C, cx, grid);
  std::lock_guard<std::mutex> order(g_bn_order);
  launch_dep(bn_sums_kernel<1>, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(dy),
             static_cast<const __nv_bfloat16*>(x), static_cast<const uint8_t*>(mask), stats, acc, M,
             C, cx);
  launch_dep(bn_bwd_apply_kernel, grid, 256, 0, s, static_cast<const __nv_bfloat16*>(dy),
             static_cast<const __nv_bfloat16*>(x), static_cast<const uint8_t*>(mask), stats, acc,
             static_cast<const __nv_bfloat16*>(gamma), static_cast<__nv_bfloat16*>(dx),
             static_cast<__nv_bfloat16*>(dres), M, C, cx);
  launch_dep(bn_param_grad_kernel, (C + 127) / 128, 128, 0, s, acc,
             static_cast<__nv_bfloat16*>(dgamma), static_cast<__nv_bfloat16*>(dbeta), C, acc_g,
             acc_b);
  return (int)cudaGetLastError();
}

extern "C" int nkb_maxpool3x3s2_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C,
                                    void* stream) {
  if (C % 8) return -3;
  const int Ho = (H + 2 - 3) / 2 + 1, Wo = (W + 2 - 3) / 2 + 1;
  launch_dep(maxpool_fwd_kernel, conv_grid((long long)N * Ho * Wo * (C / 8), 256), 256, 0,
             static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x),
             static_cast<__nv_bfloat16*>(y), static_cast<uint8_t*>(idx), N, H, W, C, Ho, Wo);
  return (int)cudaGetLastError();
}

extern "C" int nkb_maxpool3x3s2_bwd(const void* dy, const void* idx, void* dx, int N, int H, int W,
                                    int C, void* stream) {
  if (C % 8) return -3;
  const int Ho = (H + 2 - 3) / 2 + 1, Wo = (W + 2 - 3) / 2 + 1;
  const long long quads = (long long)N * ((H + 1) / 2) * ((W + 1) / 2) * (C / 8);
  launch_dep(maxpool_bwd_kernel, conv_grid(quads, 256), 256, 0, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(dy), static_cast<const uint8_t*>(idx),
             static_cast<__nv_bfloat16*>(dx), N, H, W, C, Ho, Wo);
  return (int)cudaGetLastError();
}

extern "C" int nkb_avgpool_fwd(const void* x, void* y, int N, int HW, int C, void* stream) {
  if (C % 8) return -3;
  launch_dep(avgpool_fwd_kernel, conv_grid((long long)N * (C / 8), 256), 256, 0,
             static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(x),
             static_cast<__nv_bfloat16*>(y), N, HW, C);
  return (int)cudaGetLastError();
}

extern "C" int nkb_avgpool_bwd(const void* dy, void* dx, int N, int HW, int C, void* stream) {
  if (C % 8) return -3;
  launch_dep(avgpool_bwd_kernel, conv_grid((long long)N * HW * (C / 8), 256), 256, 0,
             static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(dy),
             static_cast<__nv_bfloat16*>(dx), N, HW, C);
  return (int)cudaGetLastError();
}

NKB_DEFINE_BOUNDS_GETTER(conv)

#ifdef NKB_DEBUG_BOUNDS
// Exercises the reporting path of the debug build without touching memory: one failing
// check (index 5 of an extent of 4) is evaluated and nothing is accessed.
namespace nkb {
__global__ void bounds_selftest_kernel(int* sink) {
  if (NKB_IN_BOUNDS(5, 4)) *sink = 1;
}
}  // namespace nkb
extern "C" int nkb_debug_bounds_selftest(int* sink, void* stream) {
  nkb::bounds_selftest_kernel<<<1, 1, 0, static_cast<cudaStream_t>(stream)>>>(sink);
  return (int)cudaGetLastError();
}
#endif
