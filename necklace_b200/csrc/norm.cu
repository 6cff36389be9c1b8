// LayerNorm / RMSNorm forward and backward for bf16 activations (fp32 math).
//
// One warp owns a row and keeps it in registers, so the forward reads x once and
// writes y once; the backward reads dy and x once and writes dx once.  Weight /
// bias gradients are column sums produced by nkb_colsum into an fp32 scratch row.
// These replace torch.nn.LayerNorm / RMSNorm calls in the transformer configs;
// the reference itself has no norm kernel.
#include "ptx.cuh"
#include "nkb_api.h"

namespace nkb {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// NCH chunks of 256 elements (32 lanes x 8 bf16) cover a row of C <= NCH*256.  Bound by memory for wide
// rows, where value by value it took 64 % of the issue slots; in packed pairs 8192 x 1024 6.9 -> 6.2 us,
// 4096 x 4096 16.4 -> 13.2, 4001 x 5120 23.4 -> 17.7; 333 x 1024 2.7.
template <int NCH>
__global__ void __launch_bounds__(128)
norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                const __nv_bfloat16* __restrict__ b, __nv_bfloat16* __restrict__ y,
                float* __restrict__ stats, int rows, int C, float eps, int rms) {
  if (!grid_dep_begin()) return;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const uint4* xp = reinterpret_cast<const uint4*>(x + (long long)row * C);
  uint4 xv[NCH];
  f32x2_t sum2 = f2_pack(0.f, 0.f), var2 = sum2;
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int e = c * 256 + lane * 8;
    if (e < C) {
      xv[c] = ld_nc_v4(xp + c * 32 + lane);
      uint32_t u[4] = {xv[c].x, xv[c].y, xv[c].z, xv[c].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) sum2 = f2_add(sum2, f2_from_bf16x2(u[j]));
    }
  }
  float lo, hi, mean = 0.f;
  f2_unpack(sum2, lo, hi);
  if (!rms) mean = warp_sum(lo + hi) / C;
  const f32x2_t nm2 = f2_pack(-mean, -mean);
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int e = c * 256 + lane * 8;
    if (e < C) {
      uint32_t u[4] = {xv[c].x, xv[c].y, xv[c].z, xv[c].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const f32x2_t d = f2_add(f2_from_bf16x2(u[j]), nm2);
        var2 = f2_fma(d, d, var2);
      }
    }
  }
  f2_unpack(var2, lo, hi);
  const float var = warp_sum(lo + hi) / C;
  const float rstd = rsqrtf(var + eps);
  const f32x2_t rs2 = f2_pack(rstd, rstd);
  if (lane == 0 && stats) {
    stats[2 * row] = mean;
    stats[2 * row + 1] = rstd;
  }
  uint4* yp = reinterpret_cast<uint4*>(y + (long long)row * C);
  const uint4* wp = reinterpret_cast<const uint4*>(w);
  const uint4* bp = reinterpret_cast<const uint4*>(b);
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int e = c * 256 + lane * 8;
    if (e < C) {
      uint4 wv = __ldg(wp + c * 32 + lane);
      uint4 bv = make_uint4(0, 0, 0, 0);
      if (b) bv = __ldg(bp + c * 32 + lane);
      uint32_t u[4] = {xv[c].x, xv[c].y, xv[c].z, xv[c].w};
      uint32_t wu[4] = {wv.x, wv.y, wv.z, wv.w};
      uint32_t bu[4] = {bv.x, bv.y, bv.z, bv.w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const f32x2_t h = f2_mul(f2_add(f2_from_bf16x2(u[j]), nm2), rs2);
        o[j] = f2_to_bf16x2(f2_fma(h, f2_from_bf16x2(wu[j]), f2_from_bf16x2(bu[j])));
      }
      yp[c * 32 + lane] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

template <int NCH>
__global__ void __launch_bounds__(128)
norm_bwd_dx_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                   const __nv_bfloat16* __restrict__ w, const float* __restrict__ stats,
                   __nv_bfloat16* __restrict__ dx, int rows, int C, int rms,
                   const __nv_bfloat16* __restrict__ dres) {
  if (!grid_dep_begin()) return;
  // dres (optional): gradient that reaches x along the residual path; added here so that no
  // separate accumulation kernel runs
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const float mean = rms ? 0.f : stats[2 * row];
  const float rstd = stats[2 * row + 1];
  const uint4* xp = reinterpret_cast<const uint4*>(x + (long long)row * C);
  const uint4* gp = reinterpret_cast<const uint4*>(dy + (long long)row * C);
  const uint4* rp = reinterpret_cast<const uint4*>(dres + (dres ? (long long)row * C : 0));
  const uint4* wp = reinterpret_cast<const uint4*>(w);
  // dyw (dy*w) and xhat kept as packed bf16? keep fp32-exact by recomputing from
  // the cached raw bf16 inputs instead.
  uint4 xv[NCH], gv[NCH];
  float s1 = 0.f, s2 = 0.f;  // sum(dy*w), sum(dy*w*xhat)
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int e = c * 256 + lane * 8;
    if (e < C) {
      xv[c] = ld_nc_v4(xp + c * 32 + lane);
      gv[c] = ld_nc_v4(gp + c * 32 + lane);
      uint4 wv = __ldg(wp + c * 32 + lane);
      uint32_t xu[4] = {xv[c].x, xv[c].y, xv[c].z, xv[c].w};
      uint32_t gu[4] = {gv[c].x, gv[c].y, gv[c].z, gv[c].w};
      uint32_t wu[4] = {wv.x, wv.y, wv.z, wv.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 xf = unpack_bf16x2(xu[j]), gf = unpack_bf16x2(gu[j]), wf = unpack_bf16x2(wu[j]);
        float a0 = gf.x * wf.x, a1 = gf.y * wf.y;
        s1 += a0 + a1;
        s2 += a0 * (xf.x - mean) * rstd + a1 * (xf.y - mean) * rstd;
      }
    }
  }
  s1 = rms ? 0.f : warp_sum(s1) / C;
  s2 = warp_sum(s2) / C;
  uint4* op = reinterpret_cast<uint4*>(dx + (long long)row * C);
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    const int e = c * 256 + lane * 8;
    if (e < C) {
      uint4 wv = __ldg(wp + c * 32 + lane);
      uint4 rv = make_uint4(0, 0, 0, 0);
      if (dres) rv = ld_nc_v4(rp + c * 32 + lane);
      uint32_t xu[4] = {xv[c].x, xv[c].y, xv[c].z, xv[c].w};
      uint32_t gu[4] = {gv[c].x, gv[c].y, gv[c].z, gv[c].w};
      uint32_t wu[4] = {wv.x, wv.y, wv.z, wv.w};
      uint32_t ru[4] = {rv.x, rv.y, rv.z, rv.w};
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 xf = unpack_bf16x2(xu[j]), gf = unpack_bf16x2(gu[j]), wf = unpack_bf16x2(wu[j]);
        float2 rf = unpack_bf16x2(ru[j]);
        float h0 = (xf.x - mean) * rstd, h1 = (xf.y - mean) * rstd;
        o[j] = pack_bf16x2(rstd * (gf.x * wf.x - s1 - h0 * s2) + rf.x,
                           rstd * (gf.y * wf.y - s1 - h1 * s2) + rf.y);
      }
      op[c * 32 + lane] = make_uint4(o[0], o[1], o[2], o[3]);
    }
  }
}

// The whole backward in one pass: dx (+ dres) and the weight / bias gradients, which are sums
// over the rows of the same dy and x.  A thread owns 8 fixed columns, so its share of those
// sums stays in 16 registers over all rows of the CTA; `tpr` threads (the row's columns / 8,
// whole warps) form a group that takes ROWS rows at a time, with the next ones' loads in
// flight, and meets once per batch to add up the two row sums.  A CTA has as many groups
// as fit 512 threads, one CTA per SM: each adds its columns to the fp32 accumulator once
// and the last one (ticket) writes the bf16 gradients and leaves both at zero.
// Bound by memory: dy, x, dres in, dx out.  With a kernel for dx and one for the column sums, which
// read dy and x again: 8192 x 1024 15.6 + 12.8 us, 4096 x 4096 47.5 + 32.1 us, 512 x 256 2.1 + 4.8 us.
// In one, the 41 instructions per value set the pace (48 % of the issue slots with a quarter of the
// warps); with packed pairs, sums that halve what a lane carries at every exchange and the two factors
// kept between their uses: 8192 x 1024 21.0 -> 16.7 us, 4096 x 4096 41.6 -> 30.3, 4001 x 5120
// 75.3 -> 70.8, 512 x 256 6.0.
constexpr int NB_MAX_C = 8192;
__device__ __forceinline__ void nb_red_add_v4(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}
// The warp's sums of s1 and s2 of every row go to out[row * pitch] (x, y).  Every exchange halves
// the values that a lane still carries: 6 shuffles for two rows, where one sum after the other
// takes 20.
template <int ROWS>
__device__ __forceinline__ void nb_warp_sums(const float* s1, const float* s2, int lane, float2* out,
                                             int pitch) {
  static_assert(ROWS == 1 || ROWS == 2, "rows per batch");
  float a, b;  // s1 and s2 of the lane's row
  if constexpr (ROWS == 2) {
    const bool up = lane & 16;  // lanes 16 and up take the second row
    a = (up ? s1[1] : s1[0]) + __shfl_xor_sync(0xffffffffu, up ? s1[0] : s1[1], 16);
    b = (up ? s2[1] : s2[0]) + __shfl_xor_sync(0xffffffffu, up ? s2[0] : s2[1], 16);
  } else {
    a = s1[0];
    b = s2[0];
  }
  const bool second = lane & 8;  // of the two sums
  float v = (second ? b : a) + __shfl_xor_sync(0xffffffffu, second ? a : b, 8);
  if constexpr (ROWS == 1) v += __shfl_xor_sync(0xffffffffu, v, 16);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  if ((lane & 7) == 0 && (ROWS == 2 || lane < 16))
    reinterpret_cast<float*>(out + (ROWS == 2 ? lane >> 4 : 0) * pitch)[second] = v;
}
template <int THREADS, int ROWS>
__global__ void __launch_bounds__(THREADS, 1)
norm_bwd_all_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
                    const __nv_bfloat16* __restrict__ w, const float* __restrict__ stats,
                    __nv_bfloat16* __restrict__ dx, const __nv_bfloat16* __restrict__ dres,
                    int rows, int C, int rms, int tpr, float* __restrict__ acc,
                    int* __restrict__ ticket, __nv_bfloat16* __restrict__ dw,
                    __nv_bfloat16* __restrict__ db, int accum_w, int accum_b) {
  if (!grid_dep_begin()) return;
  extern __shared__ __align__(16) float nb_smem[];
  // [2 buffers][warps][ROWS] row sums, then [threads][16] column sums of the groups
  float2* part = reinterpret_cast<float2*>(nb_smem);
  const int warps = blockDim.x >> 5;
  const int groups = blockDim.x / tpr, wpg = tpr >> 5;
  const int grp = threadIdx.x / tpr, t = threadIdx.x - grp * tpr;
  const int lane = threadIdx.x & 31, wg = t >> 5;
  const int col = t * 8;
  const bool on = col < C;
  const float inv_c = 1.f / (float)C;
  f32x2_t wf[4], sw2[4], sb2[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) wf[j] = sw2[j] = sb2[j] = f2_pack(0.f, 0.f);
  if (on) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(w + col));
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) wf[j] = f2_from_bf16x2(u[j]);
  }
  int buf = 0;
  const int step = gridDim.x * groups * ROWS;
  uint4 xv[ROWS], gv[ROWS], rv[ROWS];
  float mean[ROWS], rstd[ROWS];
  auto fetch = [&](int row0, uint4* xo, uint4* go, uint4* ro, float* mo, float* so) {
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      xo[r] = go[r] = ro[r] = make_uint4(0, 0, 0, 0);
      mo[r] = so[r] = 0.f;
      if (row0 + r < rows) {
        const float2 st = __ldg(reinterpret_cast<const float2*>(stats) + row0 + r);
        mo[r] = rms ? 0.f : st.x;
        so[r] = st.y;
        if (on) {
          const long long off = (long long)(row0 + r) * C + col;
          xo[r] = ld_nc_v4(x + off);
          go[r] = ld_nc_v4(dy + off);
          if (dres) ro[r] = ld_nc_v4(dres + off);
        }
      }
    }
  };
  int row0 = (blockIdx.x * groups + grp) * ROWS;
  if (row0 < rows) fetch(row0, xv, gv, rv, mean, rstd);
  for (; row0 < rows; row0 += step, buf ^= 1) {
    uint4 xn[ROWS], gn[ROWS], rn[ROWS];
    float mn[ROWS], sn[ROWS];
    fetch(row0 + step, xn, gn, rn, mn, sn);  // the next batch is on its way meanwhile
    float2* mine = part + (size_t)(buf * warps + grp * wpg) * ROWS;
    // dy w and the normalised x of pair j of row r; kept between the two uses where there are
    // registers for it (the form with 64 of them spilled: 4001 x 5120 took 78 us for 71)
    constexpr bool KEEP = THREADS <= 512;
    f32x2_t ka[KEEP ? ROWS : 1][4], kh[KEEP ? ROWS : 1][4];
    auto norm2 = [&](int r, uint32_t xu) {
      return f2_mul(f2_add(f2_from_bf16x2(xu), f2_pack(-mean[r], -mean[r])),
                    f2_pack(rstd[r], rstd[r]));
    };
    float s1[ROWS], s2[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      const uint32_t xu[4] = {xv[r].x, xv[r].y, xv[r].z, xv[r].w};
      const uint32_t gu[4] = {gv[r].x, gv[r].y, gv[r].z, gv[r].w};
      f32x2_t t1 = f2_pack(0.f, 0.f), t2 = t1;
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // columns behind the last one have dy = w = 0
        const f32x2_t g = f2_from_bf16x2(gu[j]);
        const f32x2_t h = norm2(r, xu[j]), a = f2_mul(g, wf[j]);
        t1 = f2_add(t1, a);
        t2 = f2_fma(a, h, t2);
        sw2[j] = f2_fma(g, h, sw2[j]);
        sb2[j] = f2_add(sb2[j], g);
        if constexpr (KEEP) {
          ka[r][j] = a;
          kh[r][j] = h;
        }
      }
      float lo, hi;
      f2_unpack(t1, lo, hi);
      s1[r] = lo + hi;
      f2_unpack(t2, lo, hi);
      s2[r] = lo + hi;
    }
    nb_warp_sums<ROWS>(s1, s2, lane, mine + wg, wpg);
    // one meeting per batch: the next batch writes the other buffer
    if (wpg > 1) asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "r"(tpr) : "memory");
    else __syncwarp();
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      float m1 = 0.f, m2 = 0.f;
      for (int k = 0; k < wpg; ++k) {
        const float2 p = mine[r * wpg + k];
        m1 += p.x;
        m2 += p.y;
      }
      m1 = rms ? 0.f : -m1 * inv_c;
      m2 *= -inv_c;
      if (on && row0 + r < rows) {
        const uint32_t ru[4] = {rv[r].x, rv[r].y, rv[r].z, rv[r].w};
        if (!KEEP)  // (the compiler would keep them all the same)
          asm volatile("" : "+r"(xv[r].x), "+r"(xv[r].y), "+r"(xv[r].z), "+r"(xv[r].w),
                            "+r"(gv[r].x), "+r"(gv[r].y), "+r"(gv[r].z), "+r"(gv[r].w));
        const uint32_t xu[4] = {xv[r].x, xv[r].y, xv[r].z, xv[r].w};
        const uint32_t gu[4] = {gv[r].x, gv[r].y, gv[r].z, gv[r].w};
        const f32x2_t n1 = f2_pack(m1, m1), n2 = f2_pack(m2, m2), rs = f2_pack(rstd[r], rstd[r]);
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const f32x2_t h = KEEP ? kh[KEEP ? r : 0][j] : norm2(r, xu[j]);
          const f32x2_t a = KEEP ? ka[KEEP ? r : 0][j] : f2_mul(f2_from_bf16x2(gu[j]), wf[j]);
          o[j] = f2_to_bf16x2(f2_fma(rs, f2_fma(h, n2, f2_add(a, n1)), f2_from_bf16x2(ru[j])));
        }
        *reinterpret_cast<uint4*>(dx + (long long)(row0 + r) * C + col) =
            make_uint4(o[0], o[1], o[2], o[3]);
      }
      xv[r] = xn[r]; gv[r] = gn[r]; rv[r] = rn[r];
      mean[r] = mn[r]; rstd[r] = sn[r];
    }
  }
  float sw[8], sb[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    f2_unpack(sw2[j], sw[2 * j], sw[2 * j + 1]);
    f2_unpack(sb2[j], sb[2 * j], sb[2 * j + 1]);
  }
  // column sums: groups of the CTA through shared memory, then one vector reduction per four
  if (groups > 1) {
    __syncthreads();
    if (grp) {
      float4* o = reinterpret_cast<float4*>(nb_smem) + (size_t)((grp - 1) * tpr + t) * 4;
      o[0] = make_float4(sw[0], sw[1], sw[2], sw[3]);
      o[1] = make_float4(sw[4], sw[5], sw[6], sw[7]);
      o[2] = make_float4(sb[0], sb[1], sb[2], sb[3]);
      o[3] = make_float4(sb[4], sb[5], sb[6], sb[7]);
    }
    __syncthreads();
    if (grp == 0)
      for (int k = 0; k + 1 < groups; ++k) {
        const float* o = nb_smem + (size_t)(k * tpr + t) * 16;
#pragma unroll
        for (int j = 0; j < 8; ++j) { sw[j] += o[j]; sb[j] += o[8 + j]; }
      }
  }
  if (grp == 0 && on) {
    nb_red_add_v4(acc + col, sw[0], sw[1], sw[2], sw[3]);
    nb_red_add_v4(acc + col + 4, sw[4], sw[5], sw[6], sw[7]);
    if (db) {
      nb_red_add_v4(acc + C + col, sb[0], sb[1], sb[2], sb[3]);
      nb_red_add_v4(acc + C + col + 4, sb[4], sb[5], sb[6], sb[7]);
    }
  }
  __shared__ int last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  // the sums lie in L2 (every CTA's reductions are fenced before its ticket); four columns of
  // both per thread
  for (int c = threadIdx.x * 4; c < C; c += blockDim.x * 4) {
    float4 a = __ldcg(reinterpret_cast<const float4*>(acc + c)), b = a;
    if (db) b = __ldcg(reinterpret_cast<const float4*>(acc + C + c));
    *reinterpret_cast<float4*>(acc + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    if (accum_w) {
      a.x += __bfloat162float(dw[c]);     a.y += __bfloat162float(dw[c + 1]);
      a.z += __bfloat162float(dw[c + 2]); a.w += __bfloat162float(dw[c + 3]);
    }
    dw[c] = __float2bfloat16(a.x);     dw[c + 1] = __float2bfloat16(a.y);
    dw[c + 2] = __float2bfloat16(a.z); dw[c + 3] = __float2bfloat16(a.w);
    if (db) {
      *reinterpret_cast<float4*>(acc + C + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (accum_b) {
        b.x += __bfloat162float(db[c]);     b.y += __bfloat162float(db[c + 1]);
        b.z += __bfloat162float(db[c + 2]); b.w += __bfloat162float(db[c + 3]);
      }
      db[c] = __float2bfloat16(b.x);     db[c + 1] = __float2bfloat16(b.y);
      db[c + 2] = __float2bfloat16(b.z); db[c + 3] = __float2bfloat16(b.w);
    }
  }
  if (threadIdx.x == 0) *ticket = 0;
}

template <int THREADS, int ROWS>
static int launch_bwd_all(const void* dy, const void* x, const void* w, const float* stats,
                          void* dx, const void* dres, int rows, int C, int rms, float* acc,
                          int* ticket, void* dw, void* db, int accum_w, int accum_b,
                          cudaStream_t s) {
  const int tpr = (C / 8 + 31) / 32 * 32;
  int groups = THREADS / tpr;
  const int want = (rows + ROWS - 1) / ROWS;      // batches of rows
  if (groups > 15) groups = 15;                   // one named barrier each
  // few rows: spread over the SMs first, but not below four warps (the last CTA writes C columns)
  while (groups > 1 && groups * 74 > want && groups * tpr > 128) groups >>= 1;
  int grid = (want + groups - 1) / groups;
  if (grid > 148) grid = 148;
  const int threads = groups * tpr;
  size_t smem = sizeof(float2) * 2 * (threads / 32) * ROWS;
  const size_t cols = groups > 1 ? sizeof(float) * 16 * (size_t)(groups - 1) * tpr : 0;
  if (cols > smem) smem = cols;
  launch_dep(norm_bwd_all_kernel<THREADS, ROWS>, grid, threads, smem, s,
             static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x),
             static_cast<const __nv_bfloat16*>(w), stats, static_cast<__nv_bfloat16*>(dx),
             static_cast<const __nv_bfloat16*>(dres), rows, C, rms, tpr, acc, ticket,
             static_cast<__nv_bfloat16*>(dw), static_cast<__nv_bfloat16*>(db), accum_w, accum_b);
  return (int)cudaGetLastError();
}

// Column sums.  Block = 32 x 8 threads: a lane owns 8 adjacent columns (one 16-byte piece
// per row), the 8 warps take interleaved rows; grid = (ceil(C/256), row_splits).
//
// Plain sums (bias gradients): a thread loads COLSUM_UNROLL rows before it adds the first, as pairs:
// 12 instructions for 8 values (through the ring, one by one: 8192 x 1024 6.5 -> 5.8 us, 8192 x 4096
// 14.5 -> 10.5, 2313 x 3072 6.1 -> 5.4; 512 x 256 3.9 -> 4.3).
//
// With the norm input (NORM): each thread streams its pieces through a private ring of COLSUM_RING
// shared-memory slots filled by cp.async (no registers held while in flight, no barriers: a thread
// only reads what it copied itself), so a CTA keeps COLSUM_RING x 8 KB in flight; plain register
// loads kept only ~1 load per warp outstanding at 2.4 TB/s.
constexpr int COLSUM_RING = 8;
constexpr int COLSUM_UNROLL = 8;  // rows in flight per thread, and per warp at least
// the ring, or the reduction buffer alone
template <bool NORM>
constexpr int colsum_smem_bytes() {
  return NORM ? 2 * COLSUM_RING * 256 * 16 : 8 * (256 + 8) * 4;
}
__device__ __forceinline__ void colsum_cp16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc)
               : "memory");
}
template <bool NORM>
__global__ void __launch_bounds__(256)
colsum_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x,
              const float* __restrict__ stats, float* __restrict__ acc, int rows, int C,
              long long ld, int rms, int* __restrict__ tickets, __nv_bfloat16* __restrict__ out,
              int accumulate) {
  if (!grid_dep_begin()) return;
  // ring slots [which: dy | x][slot][thread] (16 bytes each); the reduction buffer reuses it
  extern __shared__ __align__(16) uint8_t colsum_smem[];  // colsum_smem_bytes<NORM>(), dynamic
  uint4 (*ring)[COLSUM_RING][256] = reinterpret_cast<uint4 (*)[COLSUM_RING][256]>(colsum_smem);
  float (*sh)[256 + 8] = reinterpret_cast<float (*)[256 + 8]>(colsum_smem);
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int col = blockIdx.x * 256 + lane * 8;
  float a[8], b[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = b[k] = 0.f;
  const bool vec = (col + 8 <= C) && ((ld & 7) == 0) &&
                   ((reinterpret_cast<uintptr_t>(dy) & 15) == 0) &&
                   (!NORM || (reinterpret_cast<uintptr_t>(x) & 15) == 0);
  const int stride = gridDim.y * 8;
  const int r0 = blockIdx.y * 8 + wy;
  if (!NORM && col < C && vec) {
    f32x2_t t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) t[j] = f2_pack(0.f, 0.f);
    for (long long r = r0; r < rows; r += COLSUM_UNROLL * stride) {
      uint4 v[COLSUM_UNROLL];
#pragma unroll
      for (int u = 0; u < COLSUM_UNROLL; ++u) {
        v[u] = make_uint4(0, 0, 0, 0);
        if (r + u * stride < rows) v[u] = ld_nc_v4(dy + (r + u * stride) * ld + col);
      }
#pragma unroll
      for (int u = 0; u < COLSUM_UNROLL; ++u) {
        t[0] = f2_add(t[0], f2_from_bf16x2(v[u].x));
        t[1] = f2_add(t[1], f2_from_bf16x2(v[u].y));
        t[2] = f2_add(t[2], f2_from_bf16x2(v[u].z));
        t[3] = f2_add(t[3], f2_from_bf16x2(v[u].w));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) f2_unpack(t[j], b[2 * j], b[2 * j + 1]);
  } else if (NORM && col < C && vec) {
    const int n = r0 < rows ? (rows - r0 + stride - 1) / stride : 0;  // rows of this thread
    auto issue = [&](int k) {
      if (k < n) {
        const long long off = (long long)(r0 + (long long)k * stride) * ld + col;
        colsum_cp16(&ring[0][k % COLSUM_RING][threadIdx.x], dy + off);
        colsum_cp16(&ring[1][k % COLSUM_RING][threadIdx.x], x + off);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");  // one group per step, empty or not
    };
#pragma unroll
    for (int k = 0; k < COLSUM_RING; ++k) issue(k);
    for (int k = 0; k < n; ++k) {
      asm volatile("cp.async.wait_group %0;" ::"n"(COLSUM_RING - 1) : "memory");
      const uint4 gu = ring[0][k % COLSUM_RING][threadIdx.x];
      const uint32_t w[4] = {gu.x, gu.y, gu.z, gu.w};
      const uint4 xu = ring[1][k % COLSUM_RING][threadIdx.x];
      const uint32_t v[4] = {xu.x, xu.y, xu.z, xu.w};
      const long long rr = r0 + (long long)k * stride;
      const float mean = rms ? 0.f : stats[2 * rr];
      const float rstd = stats[2 * rr + 1];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = unpack_bf16x2(w[j]), xf = unpack_bf16x2(v[j]);
        b[2 * j] += f.x;
        b[2 * j + 1] += f.y;
        a[2 * j] += f.x * (xf.x - mean) * rstd;
        a[2 * j + 1] += f.y * (xf.y - mean) * rstd;
      }
      issue(k + COLSUM_RING);  // refill the slot just read
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  } else if (col < C) {
    for (int r = r0; r < rows; r += stride) {
      float g[8], xv[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        g[k] = (col + k < C) ? __bfloat162float(dy[(long long)r * ld + col + k]) : 0.f;
        xv[k] = (NORM && col + k < C) ? __bfloat162float(x[(long long)r * ld + col + k]) : 0.f;
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) b[k] += g[k];
      if (NORM) {
        const float mean = rms ? 0.f : stats[2 * r];
        const float rstd = stats[2 * r + 1];
#pragma unroll
        for (int k = 0; k < 8; ++k) a[k] += g[k] * (xv[k] - mean) * rstd;
      }
    }
  }
  for (int which = 0; which < 2; ++which) {
    if (which == 0 && !NORM) continue;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 8; ++k) sh[wy][lane * 8 + k] = which == 0 ? a[k] : b[k];
    __syncthreads();
    const int c = threadIdx.x;
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += sh[i][c];
    const int gc = blockIdx.x * 256 + c;
    if (gc < C) atomicAdd(&acc[(long long)which * C + gc], s);
  }
  if (!tickets) return;
  // Fused finish: the last CTA of a column strip (ticket counter) turns the sums into bf16
  // outputs and leaves the accumulator and the counter at zero for the next call.
  __shared__ int sh_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) sh_last = (atomicAdd(&tickets[blockIdx.x], 1) == (int)gridDim.y - 1);
  __syncthreads();
  if (!sh_last) return;
  __threadfence();
  const int gc = blockIdx.x * 256 + threadIdx.x;
  if (gc < C) {
    float v = atomicExch(&acc[(long long)C + gc], 0.f);
    if (accumulate) v += __bfloat162float(out[gc]);
    out[gc] = __float2bfloat16(v);
  }
  if (threadIdx.x == 0) tickets[blockIdx.x] = 0;
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                   long long n, int accumulate) {
  if (!grid_dep_begin()) return;
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    float v = src[i];
    if (accumulate) v += __bfloat162float(dst[i]);
    dst[i] = __float2bfloat16(v);
  }
}

template <int NCH>
static int launch_fwd(const void* x, const void* w, const void* b, void* y, float* stats, int rows,
                      int C, float eps, int rms, cudaStream_t s) {
  launch_dep(norm_fwd_kernel<NCH>, (rows + 3) / 4, 128, 0, s, static_cast<const __nv_bfloat16*>(x),
             static_cast<const __nv_bfloat16*>(w), static_cast<const __nv_bfloat16*>(b),
             static_cast<__nv_bfloat16*>(y), stats, rows, C, eps, rms);
  return (int)cudaGetLastError();
}
template <int NCH>
static int launch_bwd(const void* dy, const void* x, const void* w, const float* stats, void* dx,
                      int rows, int C, int rms, const void* dres, cudaStream_t s) {
  launch_dep(norm_bwd_dx_kernel<NCH>, (rows + 3) / 4, 128, 0, s,
             static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x),
             static_cast<const __nv_bfloat16*>(w), stats, static_cast<__nv_bfloat16*>(dx), rows, C,
             rms, static_cast<const __nv_bfloat16*>(dres));
  return (int)cudaGetLastError();
}

}  // namespace nkb

using namespace nkb;

#define NKB_NCH_DISPATCH(FN, ...)                          \
  do {                                                     \
    const int nch = (C + 255) / 256;                       \
    if (nch <= 1) return FN<1>(__VA_ARGS__);               \
    if (nch <= 2) return FN<2>(__VA_ARGS__);               \
    if (nch <= 4) return FN<4>(__VA_ARGS__);               \
    if (nch <= 8) return FN<8>(__VA_ARGS__);               \
    if (nch <= 16) return FN<16>(__VA_ARGS__);             \
    if (nch <= 20) return FN<20>(__VA_ARGS__);             \
    if (nch <= 32) return FN<32>(__VA_ARGS__);             \
    return -4;                                             \
  } while (0)

extern "C" int nkb_norm_fwd(const void* x, const void* w, const void* b, void* y, float* stats,
                            int rows, int C, float eps, int rms, void* stream) {
  if (C % 8) return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  NKB_NCH_DISPATCH(launch_fwd, x, w, b, y, stats, rows, C, eps, rms, s);
}

extern "C" int nkb_norm_bwd_dx(const void* dy, const void* x, const void* w, const float* stats,
                               void* dx, int rows, int C, int rms, void* stream) {
  if (C % 8) return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  NKB_NCH_DISPATCH(launch_bwd, dy, x, w, stats, dx, rows, C, rms, nullptr, s);
}

// dx = norm backward of dy + dres (the gradient arriving along the residual connection)
extern "C" int nkb_norm_bwd_dx_res(const void* dy, const void* x, const void* w, const float* stats,
                                   void* dx, int rows, int C, int rms, const void* dres,
                                   void* stream) {
  if (C % 8) return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  NKB_NCH_DISPATCH(launch_bwd, dy, x, w, stats, dx, rows, C, rms, dres, s);
}

// dx = norm backward of dy (+ dres, may be null); dw, db (may be null) = bf16 gradients of weight
// and bias, written or added to.  acc: fp32 [2][C], ticket: one int, zero before the first call
// and left zero (calls that share them must be ordered on one stream).
extern "C" int nkb_norm_bwd_all(const void* dy, const void* x, const void* w, const float* stats,
                                void* dx, const void* dres, int rows, int C, int rms, float* acc,
                                int* ticket, void* dw, void* db, int accum_w, int accum_b,
                                void* stream) {
  if ((C % 8) || C <= 0 || C > nkb::NB_MAX_C || rows <= 0 || !acc || !ticket || !dw) return -3;
  if ((reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(x) |
       reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(dx) |
       reinterpret_cast<uintptr_t>(dres) | reinterpret_cast<uintptr_t>(acc)) & 15)
    return -3;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // more than 4096 columns: 1024 threads of 64 registers, half the rows in flight per thread
  if (C > 4096)
    return launch_bwd_all<1024, 1>(dy, x, w, stats, dx, dres, rows, C, rms, acc, ticket, dw, db,
                                   accum_w, accum_b, s);
  return launch_bwd_all<512, 2>(dy, x, w, stats, dx, dres, rows, C, rms, acc, ticket, dw, db,
                                accum_w, accum_b, s);
}

// row splits: about three CTAs per SM (64 KB of ring each; four without), and whole turns of
// COLSUM_UNROLL rows per warp
static int colsum_row_splits(int gx, int rows, int per_sm) {
  const int most = (per_sm * 148 + gx - 1) / gx, turn = 8 * nkb::COLSUM_UNROLL;
  const int turns = (int)((rows + (long long)turn * most - 1) / ((long long)turn * most));
  return (int)((rows + (long long)turn * turns - 1) / ((long long)turn * turns));
}

template <bool NORM>
static int launch_colsum(const void* dy, const void* x, const float* stats, float* acc, int rows,
                         int C, long long ld, int rms, int* tickets, void* out, int accumulate,
                         void* stream) {
  constexpr int smem = nkb::colsum_smem_bytes<NORM>();
  static bool done[64];
  if (nkb::allow_smem(nkb::colsum_kernel<NORM>, smem, done)) return -6;
  const int gx = (C + 255) / 256, gy = rows > 0 ? colsum_row_splits(gx, rows, NORM ? 3 : 4) : 1;
  launch_dep(colsum_kernel<NORM>, dim3(gx, gy), 256, smem, static_cast<cudaStream_t>(stream),
             static_cast<const __nv_bfloat16*>(dy), static_cast<const __nv_bfloat16*>(x), stats, acc,
             rows, C, ld, rms, tickets, static_cast<__nv_bfloat16*>(out), accumulate);
  return (int)cudaGetLastError();
}

extern "C" int nkb_colsum(const void* dy, const void* x, const float* stats, float* acc, int rows,
                          int C, long long ld, int rms, void* stream) {
  if ((C & 1) || (ld & 1)) return -3;
  return x ? launch_colsum<true>(dy, x, stats, acc, rows, C, ld, rms, nullptr, nullptr, 0, stream)
           : launch_colsum<false>(dy, x, stats, acc, rows, C, ld, rms, nullptr, nullptr, 0, stream);
}

// Column sums of dy straight to a bf16 output in one launch.  acc: fp32 [2][C] (the second half
// is used) and tickets: int [ceil(C/256)], both owned by the caller, zero before the first call
// and left zero by every call (calls that share them must be ordered on one stream).
extern "C" int nkb_colsum_fused(const void* dy, float* acc, int* tickets, void* out,
                                int accumulate, int rows, int C, long long ld, void* stream) {
  if ((C & 1) || (ld & 1) || !acc || !tickets || !out) return -3;
  return launch_colsum<false>(dy, nullptr, nullptr, acc, rows, C, ld, 0, tickets, out, accumulate,
                              stream);
}

extern "C" int nkb_f32_to_bf16(const float* src, void* dst, long long n, int accumulate,
                               void* stream) {
  if (n <= 0) return 0;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 8) blocks = 148 * 8;
  launch_dep(f32_to_bf16_kernel, blocks, 256, 0, static_cast<cudaStream_t>(stream), src,
             static_cast<__nv_bfloat16*>(dst), n, accumulate);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Allocation-free column sum (declared in nkb_noalloc.h).  The fp32 accumulator
// lives in the library image instead of caller-provided scratch.
#include "nkb_noalloc.h"

static __device__ __align__(256) float g_noalloc_colsum_scratch[2 * NKB_NOALLOC_MAX_COLS];

// Device address of the scratch array per device ordinal.  The array's name is only
// a host-side handle; kernels must be given the address cudaGetSymbolAddress returns
// while the owning device is current.
// Filled on the first call per device.  Two host threads making that first call at the
// same time both store the same address, so the slot is an atomic pointer (no lock needed:
// the look-up is idempotent) and readers never see a torn value.
#include <atomic>
static std::atomic<float*> g_noalloc_scratch_ptr[64];

extern "C" int nkb_colsum_bf16_noalloc(const void* dy, void* out, int rows, int C, long long ld,
                                       void* stream) {
  if (C > NKB_NOALLOC_MAX_COLS) return -4;
  if (C <= 0 || rows <= 0) return -2;
  if ((C & 1) || (ld & 1)) return -3;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return (int)e;
  if (dev < 0 || dev >= 64) return -5;
  float* acc = g_noalloc_scratch_ptr[dev].load(std::memory_order_acquire);
  if (!acc) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_colsum_scratch);
    if (e != cudaSuccess) return (int)e;
    acc = static_cast<float*>(p);
    g_noalloc_scratch_ptr[dev].store(acc, std::memory_order_release);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // only the plain-sum half [C, 2C) is used; it must start at zero for every call
  e = cudaMemsetAsync(acc + C, 0, sizeof(float) * (size_t)C, s);
  if (e != cudaSuccess) return (int)e;
  int rc = nkb_colsum(dy, nullptr, nullptr, acc, rows, C, ld, 0, stream);
  if (rc) return rc;
  return nkb_f32_to_bf16(acc + C, out, C, 0, stream);
}
