// Convolution without a gathered matrix, on tcgen05: forward, data gradient and weight gradient
// of channels-last (NHWC) bf16 tensors whose channel counts are multiples of 8.
//
// A convolution is a sum over the KH x KW taps of matrix products whose pixel operand is the
// image, shifted by the tap.  The pixels of a tile are a box of bw x bh x bn positions (width,
// height, image) with at most 128 of them, so one 4-D TMA load with 128-byte rows (64 channels)
// brings a tap's operand from where the image lies; what falls outside the image reads as
// zero, which is the padding, and a traversal stride in the tensor map does strided layers.
// Nothing is gathered through memory: the gathered matrix of a 3x3 layer is nine times the
// image and was written once and read twice per step.
//
//   forward        y[p, co]      = sum over tap, ci  x[p * s + tap - pad, ci]  w[co, tap, ci]
//   data gradient  dx[q, ci]     = sum over tap, co  dy[(q + pad - tap) / s, co]  w[co, tap, ci]
//                  for a stride s > 1 one launch per class of positions q mod s, whose taps are
//                  those that divide; the output is a strided view of dx.
//                  Each tap's product is rounded to bf16 before the taps are added in fp32: every
//                  tap is an accumulator of its own, which the epilogue adds up in registers.
//                  The gathered form rounds there because the products go through memory; here
//                  the only reason is that both forms of a layer then give the same results (one
//                  accumulator for all taps is quicker and rounds once: it moved results by
//                  0.26 % of their norm)
//   weight grad.   dw[co, tap, ci] = sum over p  dy[p, co]  x[p * s + tap - pad, ci]
//                  pixels are the contraction: boxes of at most 64 of them, both operands
//                  MN-major, the range of boxes split over all SMs, fp32 partial sums
//
// What bounds it: with 64 output channels the MMA (N = 64 costs as much as N = 128) and the nine
// reads of the image from L2, with more channels the tensor cores.  ResNet-50, 256 images of
// 224 x 224, the 19 layers that were gathered, in us: forward 2832 (gather) + about 1700 (GEMM)
// before, 1355 now; data gradient 2777 (scatter) + about 2500, now 1888 (1456 with one accumulator
// for all taps, which rounds once); weight gradient about 5000, now 1458.  Layers with few
// positions or few channels are quicker gathered: nkb_conv_route decides.
//
// Warp roles and pipeline are those of the GEMM (gemm_sm100.cu): one TMA producer thread, one
// MMA thread, eight epilogue warps, two accumulators in TMEM, one CTA per SM, tiles dealt
// round-robin.  All waits are bounded.
//
// The reference runs these layers through torch's cuDNN
// (examples/dp/mnist/pytorch/main.py).
#include "ptx.cuh"
#include "nkb_api.h"

namespace nkb {

int num_sms();
double gemm_time_us(int M, int N, int K);
int make_tmap_bf16_nd(CUtensorMap* out, const void* base, int rank, const long long* dims,
                      const long long* strides, const int* box, const int* estr);

constexpr int CV_BK = 64;
constexpr int CV_THREADS = 384;  // warps 0, 1: TMA and MMA; 2, 3 idle; 4..11 epilogue
constexpr int CV_A_BYTES = 128 * CV_BK * 2;
constexpr int CV_STG_BYTES = 2 * 16384;  // one 128 x 64 bf16 tile per epilogue group
constexpr int CV_MAX_TAPS = 64;
// setmaxnreg hand-over (data gradient); the CTA owns 384 threads x 168 registers
constexpr int CV_CTRL_REGS = 72, CV_EPI_REGS = 216;
static_assert(128 * CV_CTRL_REGS + 256 * CV_EPI_REGS <= CV_THREADS * 168, "register budget");
enum { CV_FWD = 0, CV_DGRAD = 1, CV_WGRAD = 2 };

struct ConvArgs {
  int bw, bh, bn, rows;     // box of pixel positions; rows = bw * bh * bn
  int nbw, nbh, nbn;        // boxes along width, height, images
  int W, H, N;              // extent of the pixel positions
  int stride;               // position -> coordinate of the shifted operand
  int ntaps;
  int kc;                   // channels contracted per tap (forward Cin, data gradient Cout)
  int cols;                 // output columns (forward Cout, data gradient Cin)
  int tiles_m, tiles_n;
  // weight gradient
  int cout, cin, cchunks;   // cchunks = 64-channel chunks of Cin
  int split;
  float* ws;                // fp32 [split][cout][ntaps * cin]
  int* status;
  int8_t offx[CV_MAX_TAPS], offy[CV_MAX_TAPS];  // shift of tap t
  uint8_t wtap[CV_MAX_TAPS];                    // its index in the weight
};

__device__ __forceinline__ void tma_store_4d(const CUtensorMap* m, const void* src, int x, int y,
                                             int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
// Barrier over `count` threads that also returns whether all of them say yes: the warps of an
// epilogue group leave together when a wait has run out in one of them.
__device__ __forceinline__ bool named_bar_and(int id, int count, bool yes) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %3, 0;\n\t"
      "barrier.cta.red.and.pred q, %1, %2, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(r) : "r"(id), "r"(count), "r"((uint32_t)yes) : "memory");
  return r != 0;
}
__device__ __forceinline__ void cv_fail(int* status, volatile int* abort_flag, int code) {
  *abort_flag = 1;
  if (status) atomicCAS(status, 0, code);
}
__device__ __forceinline__ void box_origin(const ConvArgs& g, int b, int& w0, int& h0, int& n0) {
  w0 = (b % g.nbw) * g.bw;
  b /= g.nbw;
  h0 = (b % g.nbh) * g.bh;
  n0 = (b / g.nbh) * g.bn;
}

template <int KIND, int BN>
struct ConvCfg {
  static constexpr int B_BYTES = BN * CV_BK * 2;
  static constexpr int STAGE = CV_A_BYTES + B_BYTES;
  static constexpr int STAGES = BN == 256 ? 4 : (BN == 128 ? 6 : 8);
  static constexpr int SMEM = STAGES * STAGE + CV_STG_BYTES + 1024 + 256;
  static constexpr uint32_t TMEM = 2 * BN;
};

template <int KIND, int BN>
__global__ void __launch_bounds__(CV_THREADS, 1)
conv_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
            const __grid_constant__ CUtensorMap tmO, const __grid_constant__ ConvArgs g) {
  using Cfg = ConvCfg<KIND, BN>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr bool A_MN = KIND == CV_WGRAD, B_MN = KIND != CV_FWD;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                              ~uintptr_t(1023));
  uint8_t* stg_base = smem + STAGES * Cfg::STAGE;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(stg_base + CV_STG_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* acc_full = empty_bar + STAGES;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      // with 64 columns each group of four warps drains every other tile by itself
      // (data gradient: both groups work on every tap)
      mbar_init(&acc_empty[a], BN == 64 && KIND != CV_DGRAD ? 4 : 8);
    }
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, Cfg::TMEM);
    tmem_relinquish();
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!grid_dep_wait()) return;
  const int boxes = g.nbw * g.nbh * g.nbn;
  const int tiles = g.tiles_m * g.tiles_n;
  const int units = KIND == CV_WGRAD ? tiles * g.split : tiles;
  const int kchunks = (g.kc + CV_BK - 1) / CV_BK;
  const int ksteps = KIND == CV_WGRAD ? g.rows / 16 : CV_BK / 16;

  // the data gradient's sums take up to 128 registers per epilogue thread
  if constexpr (KIND == CV_DGRAD)
    if (warp < 4) reg_alloc_dec<CV_CTRL_REGS>();
  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        if constexpr (KIND == CV_WGRAD) {
          const int t = u % tiles, ks = u / tiles;
          const int m0 = (t % g.tiles_m) * 128;
          const int j0 = (t / g.tiles_m) * (BN / 64);  // first (tap, channel chunk) of the tile
          const int b_lo = (int)((long long)ks * boxes / g.split);
          const int b_hi = (int)((long long)(ks + 1) * boxes / g.split);
          // parts that lie outside the matrix are not loaded: their rows and columns of the
          // accumulator are never read
          const int am = (g.cout - m0 + 63) / 64 < 2 ? 1 : 2;
          const int left = g.ntaps * g.cchunks - j0;
          const int bm = left < BN / 64 ? left : BN / 64;
          const uint32_t bytes = (uint32_t)(am + bm) * g.rows * 128;
          int sx[BN / 64], sy[BN / 64], sc[BN / 64];
#pragma unroll
          for (int j = 0; j < BN / 64; ++j) {
            const int q = j0 + j, tap = j < bm ? q / g.cchunks : 0;
            sx[j] = g.offx[tap];
            sy[j] = g.offy[tap];
            sc[j] = (q % g.cchunks) * 64;
          }
          for (int b = b_lo; b < b_hi; ++b) {
            int w0, h0, n0;
            box_origin(g, b, w0, h0, n0);
            if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
              cv_fail(g.status, abort_flag, NKB_ERR_EMPTY_WAIT);
              ok = false;
              break;
            }
            uint8_t* sA = smem + stage * Cfg::STAGE;
            uint8_t* sB = sA + CV_A_BYTES;
            mbar_expect_tx(&full_bar[stage], bytes);
            tma_load_4d(sA, &tmA, &full_bar[stage], m0, w0, h0, n0);
            if (am == 2) tma_load_4d(sA + 8192, &tmA, &full_bar[stage], m0 + 64, w0, h0, n0);
#pragma unroll
            for (int j = 0; j < BN / 64; ++j)
              if (j < bm)
                tma_load_4d(sB + j * 8192, &tmB, &full_bar[stage], sc[j], w0 * g.stride + sx[j],
                            h0 * g.stride + sy[j], n0);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
        } else {
          int w0, h0, n0;
          box_origin(g, u % g.tiles_m, w0, h0, n0);
          const int c0 = (u / g.tiles_m) * BN;
          const uint32_t bytes = (uint32_t)g.rows * 128 + Cfg::B_BYTES;
          for (int t = 0; t < g.ntaps && ok; ++t) {
            const int x = w0 * g.stride + g.offx[t], y = h0 * g.stride + g.offy[t];
            const int wt = g.wtap[t];
            for (int kb = 0; kb < kchunks; ++kb) {
              if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_flag)) {
                cv_fail(g.status, abort_flag, NKB_ERR_EMPTY_WAIT);
                ok = false;
                break;
              }
              uint8_t* sA = smem + stage * Cfg::STAGE;
              uint8_t* sB = sA + CV_A_BYTES;
              mbar_expect_tx(&full_bar[stage], bytes);
              tma_load_4d(sA, &tmA, &full_bar[stage], kb * 64, x, y, n0);
              if constexpr (KIND == CV_FWD) {
                tma_load_3d(sB, &tmB, &full_bar[stage], kb * 64, wt, c0);
              } else {
#pragma unroll
                for (int j = 0; j < BN / 64; ++j)
                  tma_load_3d(sB + j * 8192, &tmB, &full_bar[stage], c0 + j * 64, wt, kb * 64);
              }
              if (++stage == STAGES) { stage = 0; phase ^= 1; }
            }
          }
        }
      }
      grid_dep_trigger();
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(128, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      const uint64_t dA0 = umma_desc_sw128(smem_u32(smem), A_MN ? 8192 : 16, 1024);
      const uint64_t dB0 = umma_desc_sw128(smem_u32(smem) + CV_A_BYTES, B_MN ? 8192 : 16, 1024);
      int stage = 0, acc = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        // steps per accumulator, and accumulators: one per tap for the data gradient
        int nk = KIND == CV_DGRAD ? kchunks : g.ntaps * kchunks;
        const int na = KIND == CV_DGRAD ? g.ntaps : 1;
        if constexpr (KIND == CV_WGRAD) {
          const int ks = u / tiles;
          nk = (int)((long long)(ks + 1) * boxes / g.split) -
               (int)((long long)ks * boxes / g.split);
        }
        for (int a = 0; a < na && ok; ++a) {
          if (!mbar_wait(&acc_empty[acc], acc_phase ^ 1, abort_flag)) {
            cv_fail(g.status, abort_flag, NKB_ERR_ACC_FREE);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN;
          for (int i = 0; i < nk; ++i) {
            if (!mbar_wait(&full_bar[stage], phase, abort_flag)) {
              cv_fail(g.status, abort_flag, NKB_ERR_TMA_WAIT);
              ok = false;
              break;
            }
            tc_fence_after();
            const uint64_t dA = dA0 + (uint32_t)stage * (Cfg::STAGE >> 4);
            const uint64_t dB = dB0 + (uint32_t)stage * (Cfg::STAGE >> 4);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              if (KIND != CV_WGRAD || k < ksteps)
                umma_bf16_ss(d_tmem, dA + (A_MN ? k * (16 * 128 >> 4) : k * 2),
                             dB + (B_MN ? k * (16 * 128 >> 4) : k * 2), idesc,
                             (i > 0 || k > 0) ? 1u : 0u);
            umma_commit(&empty_bar[stage]);
            if (++stage == STAGES) { stage = 0; phase ^= 1; }
          }
          if (!ok) break;
          umma_commit(&acc_full[acc]);
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
      }
    }
  } else if (warp >= 4) {
    const int lane_grp = warp & 3;       // TMEM lanes 32 * lane_grp ..
    const int group = (warp - 4) >> 2;   // each group takes every other 64-column chunk
    uint8_t* gstg = stg_base + group * 16384;
    uint8_t* stg = gstg + lane_grp * 4096;
    int acc = 0;
    uint32_t acc_phase = 0;
    if constexpr (KIND == CV_DGRAD) {
      reg_alloc_inc<CV_EPI_REGS>();
      // a group's columns: 32 of the 64, or every other chunk of 64
      constexpr int NC = BN == 64 ? 32 : BN / 2;
      int odd = 0;  // two units' tiles of 64 columns alternate between the staging buffers
      for (int u = blockIdx.x; u < units; u += gridDim.x, odd ^= 1) {
        float sum[NC];
#pragma unroll
        for (int i = 0; i < NC; ++i) sum[i] = 0.f;
        bool ok = true;
        for (int t = 0; t < g.ntaps; ++t) {
          ok = ok && mbar_wait(&acc_full[acc], acc_phase, abort_flag);
          if (ok) {
            tc_fence_after();
            const uint32_t t_addr = tmem_base + (uint32_t(lane_grp * 32) << 16) + acc * BN;
#pragma unroll
            for (int q = 0; q < NC / 32; ++q) {
              const int c = BN == 64 ? group * 32 : ((q >> 1) * 2 + group) * 64 + (q & 1) * 32;
              uint32_t v[32];
              tmem_ld_32x32(t_addr + c, v);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const float2 f = unpack_bf16x2(
                    pack_bf16x2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])));
                sum[q * 32 + 2 * i] += f.x;
                sum[q * 32 + 2 * i + 1] += f.y;
              }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
          }
          if (++acc == 2) { acc = 0; acc_phase ^= 1; }
        }
        int w0, h0, n0;
        box_origin(g, u % g.tiles_m, w0, h0, n0);
        const int c0 = (u / g.tiles_m) * BN;
        const int bar = BN == 64 ? 3 : 1 + group, bar_n = BN == 64 ? 256 : 128;
        const bool issuer = lane_grp == 0 && lane == 0 && (BN > 64 || group == 0);
        uint8_t* tile = BN == 64 ? stg_base + odd * 16384 : gstg;
        // the store that used the staging tile before has read it; all warps agree to go on
        if (issuer) { if (BN == 64) tma_store_wait_read<1>(); else tma_store_wait_read<0>(); }
        if (!named_bar_and(bar, bar_n, ok)) {
          cv_fail(g.status, abort_flag, NKB_ERR_ACC_WAIT);
          break;
        }
#pragma unroll
        for (int ch = 0; ch < (BN == 64 ? 1 : BN / 128); ++ch) {
          const int col = c0 + (BN == 64 ? 0 : (ch * 2 + group) * 64);
          if (col >= g.cols) break;  // the same for all warps of the group
          if (ch) {
            if (issuer) tma_store_wait_read<0>();
            named_bar_sync(bar, bar_n);
          }
          constexpr int Q = BN == 64 ? 4 : 8;
#pragma unroll
          for (int k = 0; k < Q; ++k) {
            const float* f = sum + ch * 64 + k * 8;
            const int q = BN == 64 ? group * 4 + k : k;
            uint8_t* row = tile + lane_grp * 4096 + lane * 128;
            *reinterpret_cast<uint4*>(row + ((q ^ (lane & 7)) << 4)) =
                make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]),
                           pack_bf16x2(f[4], f[5]), pack_bf16x2(f[6], f[7]));
          }
          fence_proxy_async_smem();
          named_bar_sync(bar, bar_n);
          if (issuer) {
            tma_store_4d(&tmO, tile, col, w0, h0, n0);
            tma_store_commit();
          }
        }
      }
    } else for (int u = blockIdx.x; u < units; u += gridDim.x) {
      const bool mine = BN > 64 || acc == group;
      if (mine) {
        const bool ok = mbar_wait(&acc_full[acc], acc_phase, abort_flag);
        const uint32_t t_addr = tmem_base + (uint32_t(lane_grp * 32) << 16) + acc * BN;
        if constexpr (KIND == CV_WGRAD) {
          if (!ok) {
            cv_fail(g.status, abort_flag, NKB_ERR_ACC_WAIT);
            break;
          }
          tc_fence_after();
          const int t = u % tiles, ks = u / tiles;
          const int row0 = (t % g.tiles_m) * 128 + lane_grp * 32;
          const int j0 = (t / g.tiles_m) * (BN / 64);
          const long long ld = (long long)g.ntaps * g.cin;
          float* out = g.ws + ((long long)ks * g.cout + row0) * ld;
          const int rows_valid = g.cout - row0;
#pragma unroll 1
          for (int hc = 2 * group; hc < BN / 32; hc += (hc & 1) ? 3 : 1) {  // 32-column halves
            const int q = j0 + (hc >> 1);
            if (q >= g.ntaps * g.cchunks) break;
            const int c = (q % g.cchunks) * 64 + (hc & 1) * 32;
            uint32_t v[32];
            tmem_ld_32x32(t_addr + hc * 32, v);
            tmem_ld_wait();
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i)
              *reinterpret_cast<uint4*>(stg + lane * 128 + ((i ^ (lane & 7)) << 4)) =
                  make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            __syncwarp();
            float* dst = out + (long long)(q / g.cchunks) * g.cin + c;
            const int ch = lane & 7;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int row = i * 4 + (lane >> 3);
              if (row < rows_valid && c + ch * 4 < g.cin &&
                  NKB_IN_BOUNDS(dst - g.ws + row * ld + ch * 4 + 3, g.split * g.cout * ld))
                *reinterpret_cast<uint4*>(dst + row * ld + ch * 4) =
                    *reinterpret_cast<const uint4*>(stg + row * 128 + ((ch ^ (row & 7)) << 4));
            }
          }
        } else {
          int w0, h0, n0;
          box_origin(g, u % g.tiles_m, w0, h0, n0);
          const int c0 = (u / g.tiles_m) * BN;
          // the store of the tile before has read the staging tile; all four warps agree
          if (lane_grp == 0 && lane == 0) tma_store_wait_read<0>();
          if (!named_bar_and(1 + group, 128, ok)) {
            cv_fail(g.status, abort_flag, NKB_ERR_ACC_WAIT);
            break;
          }
          tc_fence_after();
#pragma unroll 1
          for (int ch = BN > 64 ? group : 0; ch < BN / 64; ch += 2) {
            if (c0 + ch * 64 >= g.cols) break;
            if (ch >= 2) {
              if (lane_grp == 0 && lane == 0) tma_store_wait_read<0>();
              named_bar_sync(1 + group, 128);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t v[32];
              tmem_ld_32x32(t_addr + ch * 64 + h * 32, v);
              tmem_ld_wait();
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const int q = h * 4 + i;
                *reinterpret_cast<uint4*>(stg + lane * 128 + ((q ^ (lane & 7)) << 4)) = make_uint4(
                    pack_bf16x2(__uint_as_float(v[8 * i]), __uint_as_float(v[8 * i + 1])),
                    pack_bf16x2(__uint_as_float(v[8 * i + 2]), __uint_as_float(v[8 * i + 3])),
                    pack_bf16x2(__uint_as_float(v[8 * i + 4]), __uint_as_float(v[8 * i + 5])),
                    pack_bf16x2(__uint_as_float(v[8 * i + 6]), __uint_as_float(v[8 * i + 7])));
              }
            }
            fence_proxy_async_smem();
            named_bar_sync(1 + group, 128);
            if (lane_grp == 0 && lane == 0) {
              // positions outside the image are clipped by the tensor map
              tma_store_4d(&tmO, gstg, c0 + ch * 64, w0, h0, n0);
              tma_store_commit();
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[acc]);
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag)  // copies and MMAs in flight land before their memory is released
      for (int i = 0; i < 1000; ++i) __nanosleep(1000);
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM);
  }
}

// dw = (accumulate ? dw : 0) + the sum of the partial matrices.  Four threads share a group of
// four values when there are many partial matrices: a layer with a small weight and many
// pixels has up to 148 of them and too few values to fill the machine with one thread each.
__global__ void __launch_bounds__(256)
conv_dw_reduce_kernel(const float* __restrict__ ws, int S, long long n4,
                      __nv_bfloat16* __restrict__ dw, int accumulate) {
  if (!grid_dep_begin()) return;
  __shared__ float4 sh[4][64];
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
  const long long i = (long long)blockIdx.x * 64 + tx;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < n4) {
    const float4* p = reinterpret_cast<const float4*>(ws) + i;
#pragma unroll 4
    for (int s = ty; s < S; s += 4) {
      const float4 v = p[(long long)s * n4];
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
  }
  sh[ty][tx] = a;
  __syncthreads();
  if (ty == 0 && i < n4) {
#pragma unroll
    for (int k = 1; k < 4; ++k) {
      const float4 v = sh[k][tx];
      a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
    }
    uint2* o = reinterpret_cast<uint2*>(dw) + i;
    if (accumulate) {
      const uint2 p = *o;
      const float2 x = unpack_bf16x2(p.x), y = unpack_bf16x2(p.y);
      a.x += x.x; a.y += x.y; a.z += y.x; a.w += y.y;
    }
    *o = make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
  }
}

// ------------------------------------------------------------------ host side
// Box of positions for a tile of at most 128: the fewest boxes over the W x H x N positions,
// then the widest (a row of pixels is contiguous).  Candidate extents are those that a number
// of equal parts gives; anything between two of them needs as many boxes as the larger.
static void pick_box(int W, int H, int N, int stride, int& bw, int& bh, int& bn) {
  const int lim = 256 / stride;  // a box spans at most 256 elements of the strided tensor
  long long best = -1;
  bw = bh = bn = 1;
  for (int w = W < 128 ? W : 128; w >= 1;) {
    if (w <= lim) {
      const int hmax = 128 / w;
      for (int h = H < hmax ? H : hmax; h >= 1;) {
        if (h <= lim) {
          int n = 128 / (w * h);
          if (n > N) n = N;
          const long long cost =
              (long long)((W + w - 1) / w) * ((H + h - 1) / h) * ((N + n - 1) / n);
          if (best < 0 || cost < best) { best = cost; bw = w; bh = h; bn = n; }
        }
        const int k = (H + h - 1) / h + 1, nx = (H + k - 1) / k;
        h = nx < h ? nx : h - 1;
      }
    }
    const int k = (W + w - 1) / w + 1, nx = (W + k - 1) / k;
    w = nx < w ? nx : w - 1;
  }
}

// Box for the contraction over positions: exactly 64, 48, 32 or 16 of them (whole MMA steps;
// positions outside read as zero).  A box costs its MMA steps and about half a step for the
// hand-over between producer and MMA thread.
static int pick_kbox(int W, int H, int N, int stride, int& bw, int& bh, int& bn) {
  const int lim = 256 / stride;
  long long best = -1;
  int rows = 0;
  for (int p = 64; p >= 16; p -= 16)
    for (int w = p; w >= 1; --w) {
      if (p % w || w > lim) continue;
      for (int h = p / w; h >= 1; --h) {
        if ((p / w) % h || h > lim) continue;
        const int n = p / w / h;
        const long long cost = (long long)((W + w - 1) / w) * ((H + h - 1) / h) *
                               ((N + n - 1) / n) * (p + 8);
        if (best < 0 || cost < best) { best = cost; bw = w; bh = h; bn = n; rows = p; }
      }
    }
  return rows;
}

static int tmap_pixels(CUtensorMap* m, const void* base, int C, int W, int H, int N, long long sw,
                       long long sh, long long sn, int bw, int bh, int bn, int stride) {
  const long long dims[4] = {C, W, H, N}, st[3] = {sw * 2, sh * 2, sn * 2};
  const int box[4] = {64, bw * stride, bh * stride, bn}, es[4] = {1, stride, stride, 1};
  return make_tmap_bf16_nd(m, base, 4, dims, st, box, es);
}

template <int KIND, int BN>
static int launch(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& o,
                  const ConvArgs& g, int units, cudaStream_t s) {
  auto kern = conv_kernel<KIND, BN>;
  static bool done[64];
  if (int e = allow_smem(kern, ConvCfg<KIND, BN>::SMEM, done)) return e;
  const int sms = num_sms();
  launch_dep(kern, units < sms ? units : sms, CV_THREADS, ConvCfg<KIND, BN>::SMEM, s, a, b, o, g);
  return (int)cudaGetLastError();
}

// Column tile: as wide as the columns allow; between 128 and 256 what the last round of tiles
// leaves idle decides, a round of 256 columns counted as 1.55 rounds of 128.  The weight is a
// GEMM's, not these kernels' own: fitted over 502 layers (see nkb_conv_route) a step of 256
// columns takes 1.25 times one of 128.
static int pick_bn(int tiles_m, int cols) {
  if (cols <= 64) return 64;
  if (cols <= 128) return 128;
  const int sms = num_sms();
  const long long t256 = (long long)tiles_m * ((cols + 255) / 256);
  const long long t128 = (long long)tiles_m * ((cols + 127) / 128);
  return (double)((t128 + sms - 1) / sms) / 0.68 < (double)((t256 + sms - 1) / sms) * 2 / 0.88
             ? 128 : 256;
}

template <int KIND>
static int run_pixels(ConvArgs& g, const CUtensorMap& a, const void* w, int C, int T, int Cout,
                      const CUtensorMap& o, cudaStream_t s) {
  const int BN = pick_bn(g.tiles_m, g.cols);
  g.tiles_n = (g.cols + BN - 1) / BN;
  CUtensorMap b;
  const long long dims[3] = {C, T, Cout}, st[2] = {2LL * C, 2LL * T * C};
  const int box[3] = {64, 1, KIND == CV_FWD ? BN : 64}, es[3] = {1, 1, 1};
  int rc = make_tmap_bf16_nd(&b, w, 3, dims, st, box, es);
  if (rc) return rc;
  const int units = g.tiles_m * g.tiles_n;
  if (BN == 64) return launch<KIND, 64>(a, b, o, g, units, s);
  if (BN == 128) return launch<KIND, 128>(a, b, o, g, units, s);
  return launch<KIND, 256>(a, b, o, g, units, s);
}

static bool conv_ok(int N, int H, int W, int C, int Cout, int KH, int KW, int stride, int pad) {
  return N > 0 && H > 0 && W > 0 && C > 0 && Cout > 0 && C % 8 == 0 && Cout % 8 == 0 && KH > 0 &&
         KW > 0 && KH * KW <= CV_MAX_TAPS && stride >= 1 && stride <= 8 && pad >= 0 && pad < 64 &&
         H + 2 * pad >= KH && W + 2 * pad >= KW;
}
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

static void set_boxes(ConvArgs& g, int W, int H, int N) {
  g.W = W; g.H = H; g.N = N;
  g.nbw = (W + g.bw - 1) / g.bw;
  g.nbh = (H + g.bh - 1) / g.bh;
  g.nbn = (N + g.bn - 1) / g.bn;
}

}  // namespace nkb

using namespace nkb;

// y [N,Ho,Wo,Cout] = conv(x [N,H,W,C], w [Cout, KH*KW*C]); -3: a shape or an alignment that the
// tensor maps cannot take.
extern "C" int nkb_conv_fwd(const void* x, const void* w, void* y, int N, int H, int W, int C,
                            int Cout, int KH, int KW, int stride, int pad, int* status,
                            void* stream) {
  if (!conv_ok(N, H, W, C, Cout, KH, KW, stride, pad) || !aligned16(x) || !aligned16(w) ||
      !aligned16(y))
    return -3;
  const int Ho = (H + 2 * pad - KH) / stride + 1, Wo = (W + 2 * pad - KW) / stride + 1;
  ConvArgs g{};
  pick_box(Wo, Ho, N, stride, g.bw, g.bh, g.bn);
  g.rows = g.bw * g.bh * g.bn;
  set_boxes(g, Wo, Ho, N);
  g.tiles_m = g.nbw * g.nbh * g.nbn;
  g.stride = stride;
  g.ntaps = KH * KW;
  for (int t = 0; t < g.ntaps; ++t) {
    g.offx[t] = (int8_t)(t % KW - pad);
    g.offy[t] = (int8_t)(t / KW - pad);
    g.wtap[t] = (uint8_t)t;
  }
  g.kc = C;
  g.cols = Cout;
  g.status = status;
  CUtensorMap a, o;
  int rc = tmap_pixels(&a, x, C, W, H, N, C, (long long)W * C, (long long)H * W * C, g.bw, g.bh,
                       g.bn, stride);
  if (!rc)
    rc = tmap_pixels(&o, y, Cout, Wo, Ho, N, Cout, (long long)Wo * Cout,
                     (long long)Ho * Wo * Cout, g.bw, g.bh, g.bn, 1);
  if (rc) return rc;
  return run_pixels<CV_FWD>(g, a, w, C, g.ntaps, Cout, o, static_cast<cudaStream_t>(stream));
}

// dx [N,H,W,C] from dy [N,Ho,Wo,Cout]; stride 1 or 2.  Consecutive taps meet every class of
// positions unless the window is smaller than the stride; then dx is cleared first.
extern "C" int nkb_conv_dgrad(const void* dy, const void* w, void* dx, int N, int H, int W, int C,
                              int Cout, int KH, int KW, int stride, int pad, int* status,
                              void* stream) {
  if (!conv_ok(N, H, W, C, Cout, KH, KW, stride, pad) || stride > 2 || !aligned16(dy) ||
      !aligned16(w) || !aligned16(dx))
    return -3;
  const int Ho = (H + 2 * pad - KH) / stride + 1, Wo = (W + 2 * pad - KW) / stride + 1;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int s1 = stride;
  if (KH < s1 || KW < s1) {
    cudaError_t e = cudaMemsetAsync(dx, 0, 2ull * N * H * W * C, s);
    if (e != cudaSuccess) return (int)e;
  }
  for (int ph = 0; ph < s1; ++ph)
    for (int pw = 0; pw < s1; ++pw) {
      const int Hc = (H - ph + s1 - 1) / s1, Wc = (W - pw + s1 - 1) / s1;
      if (Hc <= 0 || Wc <= 0) continue;
      ConvArgs g{};
      for (int t = 0; t < KH * KW; ++t) {
        const int oy = ph + pad - t / KW, ox = pw + pad - t % KW;
        if (oy % s1 || ox % s1) continue;
        g.offy[g.ntaps] = (int8_t)(oy / s1);
        g.offx[g.ntaps] = (int8_t)(ox / s1);
        g.wtap[g.ntaps++] = (uint8_t)t;
      }
      if (!g.ntaps) continue;
      pick_box(Wc, Hc, N, 1, g.bw, g.bh, g.bn);
      g.rows = g.bw * g.bh * g.bn;
      set_boxes(g, Wc, Hc, N);
      g.tiles_m = g.nbw * g.nbh * g.nbn;
      g.stride = 1;
      g.kc = Cout;
      g.cols = C;
      g.status = status;
      CUtensorMap a, o;
      int rc = tmap_pixels(&a, dy, Cout, Wo, Ho, N, Cout, (long long)Wo * Cout,
                           (long long)Ho * Wo * Cout, g.bw, g.bh, g.bn, 1);
      if (!rc)
        rc = tmap_pixels(&o, static_cast<__nv_bfloat16*>(dx) + ((long long)ph * W + pw) * C, C, Wc,
                         Hc, N, (long long)s1 * C, (long long)s1 * W * C, (long long)H * W * C,
                         g.bw, g.bh, g.bn, 1);
      if (rc) return rc;
      rc = run_pixels<CV_DGRAD>(g, a, w, C, KH * KW, Cout, o, s);
      if (rc) return rc;
    }
  return 0;
}

// Number of partial matrices that nkb_conv_wgrad writes for this layer (its workspace is that
// many fp32 [Cout, KH*KW*C] matrices), or -3.  The (row tile, column tile) pairs of a small
// weight are far fewer than SMs while the pixels are many: the pixel range is cut so that the
// units fill the SMs once, with at least four boxes of pixels per unit.
static int wgrad_plan(ConvArgs& g, int N, int H, int W, int C, int Cout, int KH, int KW,
                      int stride, int pad, int& BN) {
  if (!conv_ok(N, H, W, C, Cout, KH, KW, stride, pad)) return -3;
  const int Ho = (H + 2 * pad - KH) / stride + 1, Wo = (W + 2 * pad - KW) / stride + 1;
  g.rows = pick_kbox(Wo, Ho, N, stride, g.bw, g.bh, g.bn);
  set_boxes(g, Wo, Ho, N);
  g.ntaps = KH * KW;
  g.cin = C;
  g.cout = Cout;
  g.cchunks = (C + 63) / 64;
  g.stride = stride;
  const int chunks = g.ntaps * g.cchunks;
  BN = chunks <= 2 ? 128 : 256;
  g.tiles_m = (Cout + 127) / 128;
  g.tiles_n = (chunks + BN / 64 - 1) / (BN / 64);
  const int boxes = g.nbw * g.nbh * g.nbn, tiles = g.tiles_m * g.tiles_n, sms = num_sms();
  // rounds x work per round: one round when it fits, else the split with the fullest last round
  int best = 1;
  double cost = 1e30;
  for (int S = 1; S <= sms && S <= 64 + sms / tiles; ++S) {
    if (S > 1 && boxes / S < 4) break;
    const long long rounds = ((long long)tiles * S + sms - 1) / sms;
    // a partial matrix is written and read again: about the time of two boxes
    const double c = rounds * ((double)boxes / S + 2.0);
    if (c < cost * 0.98) { cost = c; best = S; }
    if (rounds > 3) break;
  }
  return best;
}

extern "C" int nkb_conv_wgrad_split(int N, int H, int W, int C, int Cout, int KH, int KW,
                                    int stride, int pad) {
  ConvArgs g{};
  int BN;
  return wgrad_plan(g, N, H, W, C, Cout, KH, KW, stride, pad, BN);
}

extern "C" int nkb_conv_wgrad(const void* x, const void* dy, void* dw, float* ws, int split, int N,
                              int H, int W, int C, int Cout, int KH, int KW, int stride, int pad,
                              int accumulate, int* status, void* stream) {
  ConvArgs g{};
  int BN;
  g.split = wgrad_plan(g, N, H, W, C, Cout, KH, KW, stride, pad, BN);
  if (g.split < 1 || g.split != split || !aligned16(x) || !aligned16(dy) || !aligned16(dw) ||
      !aligned16(ws))
    return -3;
  for (int t = 0; t < g.ntaps; ++t) {
    g.offx[t] = (int8_t)(t % KW - pad);
    g.offy[t] = (int8_t)(t / KW - pad);
  }
  g.ws = ws;
  g.status = status;
  CUtensorMap a, b;
  int rc = tmap_pixels(&a, dy, Cout, g.W, g.H, N, Cout, (long long)g.W * Cout,
                       (long long)g.H * g.W * Cout, g.bw, g.bh, g.bn, 1);
  // Positions outside the output read dy as zero, but x at their taps may lie inside the image.
  // Pixels behind the last window (a remainder of the stride) are cut off the map: no window has
  // them, so an Inf or NaN there must not meet those zeros.  (Where a window has such a pixel,
  // its channel's gradient holds an Inf or NaN in any case.)
  const int Wu = (g.W - 1) * stride + KW - pad, Hu = (g.H - 1) * stride + KH - pad;
  if (!rc)
    rc = tmap_pixels(&b, x, C, Wu < 1 ? 1 : Wu < W ? Wu : W, Hu < 1 ? 1 : Hu < H ? Hu : H, N, C,
                     (long long)W * C, (long long)H * W * C, g.bw, g.bh, g.bn, stride);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int units = g.tiles_m * g.tiles_n * g.split;
  rc = BN == 128 ? launch<CV_WGRAD, 128>(a, b, a, g, units, s)
                 : launch<CV_WGRAD, 256>(a, b, a, g, units, s);
  if (rc) return rc;
  const long long n4 = (long long)Cout * g.ntaps * C / 4;
  launch_dep(conv_dw_reduce_kernel, (unsigned)((n4 + 63) / 64), 256, 0, s, ws, g.split, n4,
             static_cast<__nv_bfloat16*>(dw), accumulate);
  return (int)cudaGetLastError();
}

// Which of a layer's three products are quicker on the image: bit 0 forward and weight gradient
// (which use one gathered matrix otherwise), bit 1 data gradient; -3 as above.
//
// The image kernels read no gathered matrix, but a tile runs through all taps and channels one
// after the other and K is not split, so a layer with few positions and a long contraction leaves
// most SMs idle, where the GEMM of the gathered form has slices: 512 -> 512, 3x3, stride 2, 8
// images of 14 x 14 take 23 + 15 + 39 us on the image (forward, weight and data gradient; the last
// in four launches, one per class of positions), 11 + 9 + 12 us gathered.  With few channels a
// step of 64 is mostly empty and a box has rows of 16 bytes: 8 -> 64, 3x3, 128 images of 56 x 56
// take 231 + 125 + 206 us on the image, 95 + 35 + 78 gathered.  With 64 channels and more and
// pixels enough the image wins: 64 -> 64, 3x3, 64 images of 28 x 28, 13 + 18 + 19 against
// 44 + 15 + 49 us.
// Times in us fitted to 502 layers (C, Cout 8 .. 1024, windows 1 .. 7, strides 1 and 2, 1 .. 256
// images): choosing by them is 0.3 % (forward and weight gradient) and 2 % (data gradient) above
// the quicker form on average; the image for all was 23 and 28 %.  The gathered form has another
// kernel and buffer, which cost the host 6 to 8 us a pass: it must win by more than that (with 4 and
// 3 us a pass of ResNet-50 over 37 images, issued eagerly, took 3 % longer than all on the image).
extern "C" int nkb_conv_route(int N, int H, int W, int C, int Cout, int KH, int KW, int stride,
                              int pad) {
  if (!conv_ok(N, H, W, C, Cout, KH, KW, stride, pad) || stride > 2) return -3;
  const int Ho = (H + 2 * pad - KH) / stride + 1, Wo = (W + 2 * pad - KW) / stride + 1;
  const int sms = num_sms(), T = KH * KW;
  const long long P = (long long)N * Ho * Wo, K = (long long)T * C;
  if (P > (1 << 30) || K > (1 << 30)) return 3;
  auto boxes = [&](int w, int h, int s) {
    int bw, bh, bn;
    pick_box(w, h, N, s, bw, bh, bn);
    return ((w + bw - 1) / bw) * ((h + bh - 1) / bh) * ((N + bn - 1) / bn);
  };
  auto rounds = [&](int tiles_m, int cols, int& BN) {
    BN = pick_bn(tiles_m, cols);
    return (int)(((long long)tiles_m * ((cols + BN - 1) / BN) + sms - 1) / sms);
  };
  // what a box of rows narrower than 128 bytes costs more, when there are many of them
  auto narrow = [](int channels, double us) { return channels < 64 ? us / channels : 0.0; };
  int BN;
  int r = rounds(boxes(Wo, Ho, stride), Cout, BN);
  double step = (0.284 + (r > 1 ? narrow(C, 3.5) : 0.0)) * (BN == 256 ? 1.25 : 1.0);
  double image = 3.1 + r * (T * ((C + 63) / 64) * step + 0.9);
  ConvArgs g{};
  const int split = wgrad_plan(g, N, H, W, C, Cout, KH, KW, stride, pad, BN);
  const int units = g.tiles_m * g.tiles_n * split;
  const int per_unit = (g.nbw * g.nbh * g.nbn + split - 1) / split;
  step = 0.56 * g.rows / 64 * (BN == 256 ? 1.0 : 0.37) + narrow(C, 1.6);
  image += 5.6 + (units + sms - 1) / sms * (per_unit * step + 1.65) +
           (double)split * Cout * K * 1.4e-6;
  const double mb = P * K * 2e-6;  // the gathered matrix, MB
  const double gather = 1.2 + mb / 1.95;
  const double gathered = gather * (mb > 2147.0 ? 2 : 1) +  // (it is not kept then)
                          gemm_time_us((int)P, Cout, (int)K) +
                          0.93 * gemm_time_us(Cout, (int)K, (int)P);
  double image_dx = 0.0;
  for (int ph = 0; ph < stride; ++ph)
    for (int pw = 0; pw < stride; ++pw) {
      const int Hc = (H - ph + stride - 1) / stride, Wc = (W - pw + stride - 1) / stride;
      int taps = 0;
      for (int t = 0; t < T; ++t)
        taps += (ph + pad - t / KW) % stride == 0 && (pw + pad - t % KW) % stride == 0;
      if (Hc <= 0 || Wc <= 0 || !taps) continue;
      r = rounds(boxes(Wc, Hc, 1), C, BN);
      // a tap's MMAs, or its way out of the accumulator
      const double mma = (Cout + 63) / 64 *
                         (0.385 * (BN == 256 ? 1.1 : 1.0) + (r > 1 ? narrow(Cout, 2.0) : 0.0));
      const double drain = 0.6 * BN / 128;
      image_dx += 3.2 + r * (taps * (mma > drain ? mma : drain) + 1.6);
    }
  const double gathered_dx = 4.9 + mb / 1.5 + gemm_time_us((int)P, (int)K, Cout);
  return (image <= gathered + 8.0 ? 1 : 0) | (image_dx <= gathered_dx + 6.0 ? 2 : 0);
}

NKB_DEFINE_WAIT_SETTER(conv)
NKB_DEFINE_BOUNDS_GETTER(convimg)
