// Bandwidth-bound kernels of the training step, written for sm_100a:
// RMSNorm / LayerNorm (+ residual add) forward and backward, rotary embedding
// (plain, multimodal-sectioned, multimodal-interleaved, vision 2-D all reduce to a
// per-token cos/sin table plus one apply kernel), SwiGLU, flat-buffer AdamW, Muon
// momentum / scale / update, EMA, gradient norm + clip, index gather/scatter for packed
// sequences, and the cross-entropy passes that follow the logits GEMM.
//
// All kernels use 16-byte vector accesses, grid-stride loops sized to the SM count and
// fp32 arithmetic on bf16 storage.  Reference behaviour: Liger RMSNorm / RoPE / SwiGLU
// (src/lmms_engine/models/qwen2/monkey_patch.py:47-118), torch.optim.AdamW
// (src/lmms_engine/train/fsdp2/fsdp2_trainer.py:202-209), the Muon update
// (src/lmms_engine/utils/muon_utils.py:159-183, 273-275), EMA
// (src/lmms_engine/utils/ema_utils.py:97-101) and foreach grad clipping
// (src/lmms_engine/utils/fsdp2_utils.py:250-289).
#include "common.cuh"

#include <cstdlib>

namespace b200 {

typedef __nv_bfloat16 bf16;

struct alignas(16) bf16x8 {
  uint32_t w[4];
};

__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
  bf16x8 u = *reinterpret_cast<const bf16x8*>(p);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 f = unpack_bf16x2(u.w[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void store8(bf16* p, const float (&v)[8]) {
  bf16x8 u;
#pragma unroll
  for (int i = 0; i < 4; ++i) u.w[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<bf16x8*>(p) = u;
}

template <int kThreads>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = (lane < kThreads / 32) ? red[lane] : 0.f;
  t = warp_sum(t);
  __syncthreads();
  return t;
}

// ------------------------------------------------------------------ RMSNorm / LayerNorm forward
// One CTA per row (H >= 1024) keeps the row in registers: H <= kThreads * 8 * kVecPerThread.
// y = (x [+ res]) * rstd * (w + w_offset);  optional res_out = x + res;  LayerNorm when `ln`.
template <int kThreads, int kVec>
__global__ void __launch_bounds__(kThreads) norm_fwd_kernel(const bf16* __restrict__ x, const bf16* __restrict__ res,
                                                            const bf16* __restrict__ w, const bf16* __restrict__ b,
                                                            bf16* __restrict__ y, bf16* __restrict__ res_out,
                                                            float* __restrict__ rstd_out, float* __restrict__ mean_out,
                                                            int rows, int H, float eps, float w_offset, int ln) {
  __shared__ float red[32];
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * H;
    float v[kVec][8];
    float s = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = (i * kThreads + threadIdx.x) * 8;
      if (c < H) {
        load8(x + base + c, v[i]);
        if (res != nullptr) {
          float r[8];
          load8(res + base + c, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] += r[j];
          // round the sum to bf16 so that the normalised row matches the stored residual stream
#pragma unroll
          for (int j = 0; j < 8; ++j) v[i][j] = __bfloat162float(__float2bfloat16(v[i][j]));
          if (res_out != nullptr) store8(res_out + base + c, v[i]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          s += v[i][j];
          s2 += v[i][j] * v[i][j];
        }
      }
    }
    float mean = 0.f;
    if (ln) {
      mean = block_sum<kThreads>(s, red) / H;
      float var = 0.f;
#pragma unroll
      for (int i = 0; i < kVec; ++i) {
        const int c = (i * kThreads + threadIdx.x) * 8;
        if (c < H) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float d = v[i][j] - mean;
            var += d * d;
          }
        }
      }
      s2 = block_sum<kThreads>(var, red);
    } else {
      s2 = block_sum<kThreads>(s2, red);
    }
    const float rstd = rsqrtf(s2 / H + eps);
    if (threadIdx.x == 0) {
      rstd_out[row] = rstd;
      if (ln && mean_out != nullptr) mean_out[row] = mean;
    }
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = (i * kThreads + threadIdx.x) * 8;
      if (c < H) {
        float wv[8], o[8];
        load8(w + c, wv);
        float bv[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (b != nullptr) load8(b + c, bv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = (v[i][j] - mean) * rstd * (wv[j] + w_offset) + bv[j];
        store8(y + base + c, o);
      }
    }
  }
}

// One warp per row for short rows (per-head QK-norm: H = 64..512, multiple of 8).
__global__ void __launch_bounds__(256) norm_fwd_warp_kernel(const bf16* __restrict__ x, const bf16* __restrict__ w,
                                                            bf16* __restrict__ y, float* __restrict__ rstd_out, int rows,
                                                            int H, float eps, float w_offset) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < rows; row += gridDim.x * wpb) {
    const size_t base = static_cast<size_t>(row) * H;
    float v[2][8];
    float s2 = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        load8(x + base + c, v[i]);
#pragma unroll
        for (int j = 0; j < 8; ++j) s2 += v[i][j] * v[i][j];
      }
    }
    s2 = warp_sum(s2);
    const float rstd = rsqrtf(s2 / H + eps);
    if (lane == 0) rstd_out[row] = rstd;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        float wv[8], o[8];
        load8(w + c, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = v[i][j] * rstd * (wv[j] + w_offset);
        store8(y + base + c, o);
      }
    }
  }
}

// ------------------------------------------------------------------ RMSNorm / LayerNorm backward
// dx = rstd * (g - xhat * mean(g * xhat) [- mean(g) for LN]) [+ dres_in], g = dy * (w + off)
// Partial dw (and db) are accumulated per CTA in registers over its rows and written to
// dw_part[blockIdx.x, H]; a second kernel reduces the partials.
template <int kThreads, int kVec>
__global__ void __launch_bounds__(kThreads)
norm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                const float* __restrict__ rstd_in, const float* __restrict__ mean_in, const bf16* __restrict__ dres_in,
                bf16* __restrict__ dx, float* __restrict__ dw_part, float* __restrict__ db_part, int rows, int H,
                float w_offset, int ln) {
  __shared__ float red[32];
  float dw[kVec][8], db[kVec][8];
#pragma unroll
  for (int i = 0; i < kVec; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[i][j] = 0.f, db[i][j] = 0.f;

  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const size_t base = static_cast<size_t>(row) * H;
    const float rstd = rstd_in[row];
    const float mean = (ln && mean_in != nullptr) ? mean_in[row] : 0.f;
    float g[kVec][8], xh[kVec][8];
    float dot = 0.f, gsum = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = (i * kThreads + threadIdx.x) * 8;
      if (c < H) {
        float dyv[8], xv[8], wv[8];
        load8(dy + base + c, dyv);
        load8(x + base + c, xv);
        load8(w + c, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[i][j] = (xv[j] - mean) * rstd;
          g[i][j] = dyv[j] * (wv[j] + w_offset);
          dw[i][j] += dyv[j] * xh[i][j];
          db[i][j] += dyv[j];
          dot += g[i][j] * xh[i][j];
          gsum += g[i][j];
        }
      }
    }
    dot = block_sum<kThreads>(dot, red) / H;
    if (ln) gsum = block_sum<kThreads>(gsum, red) / H;
    else gsum = 0.f;
#pragma unroll
    for (int i = 0; i < kVec; ++i) {
      const int c = (i * kThreads + threadIdx.x) * 8;
      if (c < H) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * (g[i][j] - xh[i][j] * dot - gsum);
        if (dres_in != nullptr) {
          float r[8];
          load8(dres_in + base + c, r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        store8(dx + base + c, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kVec; ++i) {
    const int c = (i * kThreads + threadIdx.x) * 8;
    if (c < H) {
      float* o = dw_part + static_cast<size_t>(blockIdx.x) * H + c;
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = dw[i][j];
      if (db_part != nullptr) {
        float* ob = db_part + static_cast<size_t>(blockIdx.x) * H + c;
#pragma unroll
        for (int j = 0; j < 8; ++j) ob[j] = db[i][j];
      }
    }
  }
}

__global__ void norm_bwd_warp_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x,
                                     const bf16* __restrict__ w, const float* __restrict__ rstd_in,
                                     bf16* __restrict__ dx, float* __restrict__ dw_part, int rows, int H,
                                     float w_offset) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  const int gw = blockIdx.x * wpb + (threadIdx.x >> 5);
  float dw[2][8];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[i][j] = 0.f;
  for (int row = gw; row < rows; row += gridDim.x * wpb) {
    const size_t base = static_cast<size_t>(row) * H;
    const float rstd = rstd_in[row];
    float g[2][8], xh[2][8];
    float dot = 0.f;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        float dyv[8], xv[8], wv[8];
        load8(dy + base + c, dyv);
        load8(x + base + c, xv);
        load8(w + c, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[i][j] = xv[j] * rstd;
          g[i][j] = dyv[j] * (wv[j] + w_offset);
          dw[i][j] += dyv[j] * xh[i][j];
          dot += g[i][j] * xh[i][j];
        }
      }
    }
    dot = warp_sum(dot) / H;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        float o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = rstd * (g[i][j] - xh[i][j] * dot);
        store8(dx + base + c, o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int c = (i * 32 + lane) * 8;
    if (c < H) {
      float* o = dw_part + static_cast<size_t>(gw) * H + c;
#pragma unroll
      for (int j = 0; j < 8; ++j) o[j] = dw[i][j];
    }
  }
}

// RMSNorm backward for narrow rows (per-head norms: H = 64 / 128 / 256): LPR = H / 8 lanes hold a row, a warp works on
// 32 / LPR rows at once, a block of sixteen warps leaves ONE row of dw partials (summed over its warps in shared memory),
// so the grid can fill the machine within the same partials scratch.
template <int LPR>
__global__ void norm_bwd_narrow_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                                       const float* __restrict__ rstd_in, bf16* __restrict__ dx,
                                       float* __restrict__ dw_part, int rows, float w_offset) {
  constexpr int H = LPR * 8;
  constexpr int RPW = 32 / LPR;  // rows per warp and iteration
  __shared__ float red[16][H];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int sub = lane / LPR, col = (lane % LPR) * 8;
  const int wpb = blockDim.x >> 5;
  float wv[8], dw[8];
  load8(w + col, wv);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    wv[j] += w_offset;
    dw[j] = 0.f;
  }
  for (long row0 = (static_cast<long>(blockIdx.x) * wpb + warp) * RPW; row0 < rows;
       row0 += static_cast<long>(gridDim.x) * wpb * RPW) {
    const long row = row0 + sub;
    const bool live = row < rows;
    float dyv[8], xv[8], g[8], xh[8];
    float dot = 0.f, rstd = 0.f;
    if (live) {
      const size_t base = static_cast<size_t>(row) * H + col;
      rstd = rstd_in[row];
      load8(dy + base, dyv);
      load8(x + base, xv);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        xh[j] = xv[j] * rstd;
        g[j] = dyv[j] * wv[j];
        dw[j] += dyv[j] * xh[j];
        dot += g[j] * xh[j];
      }
    }
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
    dot /= H;
    if (live) {
      float o8[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) o8[j] = rstd * (g[j] - xh[j] * dot);
      store8(dx + static_cast<size_t>(row) * H + col, o8);
    }
  }
  // lanes that hold the same columns (one per row of the warp's group), then the block's warps
#pragma unroll
  for (int o = LPR; o < 32; o <<= 1)
#pragma unroll
    for (int j = 0; j < 8; ++j) dw[j] += __shfl_xor_sync(0xffffffffu, dw[j], o);
  if (sub == 0) {
#pragma unroll
    for (int j = 0; j < 8; ++j) red[warp][col + j] = dw[j];
  }
  __syncthreads();
  for (int c = threadIdx.x; c < H; c += blockDim.x) {
    float acc = 0.f;
    for (int q = 0; q < wpb; ++q) acc += red[q][c];
    dw_part[static_cast<size_t>(blockIdx.x) * H + c] = acc;
  }
}

// Backward for rows of up to 256 VEC columns, one warp per row: a row's dy and x stay packed in registers between the sums and
// the result, no barrier separates one row from the next, and eight (sixteen) rows per SM are on their way at once.  A CTA per
// row kept two rows per SM in flight and paid up to four barriers for each: 21.9k x 1280 85 us, 4096 x 1024 23 us a call, three
// to five times what their bytes take.  A CTA leaves one row of dw (db) partials.
template <int VEC, bool LN, bool RES>
__global__ void __launch_bounds__(256, VEC <= 4 ? 2 : 1)
norm_bwd_rows_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const bf16* __restrict__ w,
                     const float* __restrict__ rstd_in, const float* __restrict__ mean_in, const bf16* __restrict__ dres_in,
                     bf16* __restrict__ dx, float* __restrict__ dw_part, float* __restrict__ db_part, int rows, int H,
                     float w_offset) {
  __shared__ float sw[LN ? 2 : 1][VEC * 256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float dw[VEC][8], db[LN ? VEC : 1][8];
#pragma unroll
  for (int i = 0; i < VEC; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dw[i][j] = 0.f;
      if (LN) db[i][j] = 0.f;
    }
  for (int row = blockIdx.x * 8 + warp; row < rows; row += gridDim.x * 8) {
    const size_t base = static_cast<size_t>(row) * H;
    const float rstd = rstd_in[row];
    const float mean = LN && mean_in != nullptr ? mean_in[row] : 0.f;
    uint4 rd[VEC], rx[VEC], rr[RES ? VEC : 1];
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        rd[i] = *reinterpret_cast<const uint4*>(dy + base + c);
        rx[i] = *reinterpret_cast<const uint4*>(x + base + c);
        if (RES) rr[i] = *reinterpret_cast<const uint4*>(dres_in + base + c);
      }
    }
    auto words = [](const uint4& u, float (&v)[8]) {
      const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
      v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
    };
    float dots[8] = {}, gsums[8] = {};   // of 256 columns each
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        float d[8], v[8], wv[8];
        words(rd[i], d);
        words(rx[i], v);
        load8(w + c, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (v[j] - mean) * rstd, g = d[j] * (wv[j] + w_offset);
          dw[i][j] += d[j] * xh;
          if (LN) db[i][j] += d[j];
          dots[i] += g * xh;
          if (LN) gsums[i] += g;
        }
      }
    }
    // the order of a CTA per row with a warp per 256 columns, which rows above 2048 columns and the forward passes have: dx
    // does not depend on which of the kernels ran (the weight gradients are summed per warp here, in another order)
    auto total = [](float (&s)[8]) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) s[i] = warp_sum(s[i]);
      return ((s[0] + s[4]) + (s[2] + s[6])) + ((s[1] + s[5]) + (s[3] + s[7]));
    };
    const float dot = total(dots) / H;
    const float gsum = LN ? total(gsums) / H : 0.f;
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
      const int c = (i * 32 + lane) * 8;
      if (c < H) {
        float d[8], v[8], wv[8], o[8];
        words(rd[i], d);
        words(rx[i], v);
        load8(w + c, wv);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xh = (v[j] - mean) * rstd, g = d[j] * (wv[j] + w_offset);
          o[j] = rstd * (g - xh * dot - gsum);
        }
        if (RES) {
          float r[8];
          words(rr[i], r);
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] += r[j];
        }
        store8(dx + base + c, o);
      }
    }
  }
  // the warps one after the other: the same sum on every run
  for (int q = 0; q < 8; ++q) {
    if (warp == q) {
#pragma unroll
      for (int i = 0; i < VEC; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int c = (i * 32 + lane) * 8 + j;
          sw[0][c] = (q == 0 ? 0.f : sw[0][c]) + dw[i][j];
          if (LN) sw[LN ? 1 : 0][c] = (q == 0 ? 0.f : sw[LN ? 1 : 0][c]) + db[LN ? i : 0][j];
        }
    }
    __syncthreads();
  }
  for (int c = threadIdx.x; c < H; c += 256) {
    dw_part[static_cast<size_t>(blockIdx.x) * H + c] = sw[0][c];
    if (LN && db_part != nullptr) db_part[static_cast<size_t>(blockIdx.x) * H + c] = sw[LN ? 1 : 0][c];
  }
}

// out[c] = sum_p part[p, c]  (fp32 -> fp32, optionally accumulating into out): 32 columns a CTA, every 32nd row a thread, in a
// fixed order.  One thread per column walked 296 rows of partials with four to eight CTAs on the chip: 11 us a call.
__global__ void __launch_bounds__(1024) colsum_kernel(const float* __restrict__ part, float* __restrict__ out, int parts, int H,
                                                      int accumulate) {
  __shared__ float sm[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < H) {
#pragma unroll 4
    for (int p = ty; p < parts; p += 32) s += part[static_cast<size_t>(p) * H + c];
  }
  sm[ty][tx] = s;
  __syncthreads();
  // row ty of the transposed tile: the 32 sums of column blockIdx.x * 32 + ty
  const float t = warp_sum(sm[tx][ty]);
  const int co = blockIdx.x * 32 + ty;
  if (tx == 0 && co < H) out[co] = accumulate ? out[co] + t : t;
}
static void colsum(const float* part, float* out, int parts, int H, int accumulate, cudaStream_t st) {
  colsum_kernel<<<(H + 31) / 32, 1024, 0, st>>>(part, out, parts, H, accumulate);
}

// Column sums of a bf16 matrix (bias gradients), fp32 inside, bf16 out.  A CTA takes 256 columns and every gridDim.y-th block
// of eight rows, four rows of a warp's loads in flight; the partials are summed by colsum_bf16_finish_kernel in a fixed order.
// Bound by reading the matrix once (the framework's reduction: 38 us for 22.4k x 1152).  Rows may be wider than N: the last
// 16-byte piece of a row may reach into its padding, which is read and dropped.
__global__ void __launch_bounds__(256) colsum_bf16_kernel(const bf16* __restrict__ x, long ld, float* __restrict__ part, long rows, int N) {
  __shared__ float sm[8][256 + 8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 256 + lane * 8;
  float acc[8] = {};
  if (c < N) {
    const long step = static_cast<long>(gridDim.y) * 8;
    long r = static_cast<long>(blockIdx.y) * 8 + warp;
    for (; r + 3 * step < rows; r += 4 * step) {
      float v[4][8];
#pragma unroll
      for (int k = 0; k < 4; ++k) load8(x + (r + k * step) * ld + c, v[k]);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += (v[0][j] + v[1][j]) + (v[2][j] + v[3][j]);
    }
    for (; r < rows; r += step) {
      float v[8];
      load8(x + r * ld + c, v);
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] += v[j];
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) sm[warp][lane * 8 + j] = acc[j];
  __syncthreads();
  const int co = blockIdx.x * 256 + threadIdx.x;
  float s = 0.f;
#pragma unroll
  for (int q = 0; q < 8; ++q) s += sm[q][threadIdx.x];
  if (co < N) part[static_cast<size_t>(blockIdx.y) * N + co] = s;
}
__global__ void __launch_bounds__(1024) colsum_bf16_finish_kernel(const float* __restrict__ part, bf16* __restrict__ out, int parts, int N) {
  __shared__ float sm[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5, c = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (c < N) {
#pragma unroll 4
    for (int p = ty; p < parts; p += 32) s += part[static_cast<size_t>(p) * N + c];
  }
  sm[ty][tx] = s;
  __syncthreads();
  const float t = warp_sum(sm[tx][ty]);
  const int co = blockIdx.x * 32 + ty;
  if (tx == 0 && co < N) out[co] = __float2bfloat16(t);
}

// ------------------------------------------------------------------ rotary embedding
// cos/sin tables [T, D] (fp32) from up to three position streams.
// mode 0: plain (pos[0]);  mode 1: sectioned M-RoPE (frequency i uses stream by section
// boundaries s0, s0+s1);   mode 2: interleaved M-RoPE (Qwen3-VL: frequency i uses stream
// i % 3 while i < 3*section[i % 3] for streams 1, 2; stream 0 otherwise).
__global__ void rope_table_kernel(const int64_t* __restrict__ pos, const float* __restrict__ inv_freq,
                                  float* __restrict__ cos_out, float* __restrict__ sin_out, int T, int half,
                                  int mode, int s0, int s1, int s2, float scaling) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= T * half) return;
  const int t = idx / half, i = idx - t * half;
  int stream = 0;
  if (mode == 1) {
    stream = (i < s0) ? 0 : (i < s0 + s1 ? 1 : 2);
  } else if (mode == 2) {
    const int m = i % 3;
    if (m == 1 && i < 3 * s1) stream = 1;
    else if (m == 2 && i < 3 * s2) stream = 2;
    else stream = 0;
  }
  const float ang = static_cast<float>(pos[static_cast<size_t>(stream) * T + t]) * inv_freq[i];
  float sn, cs;
  sincosf(ang, &sn, &cs);
  cs *= scaling;
  sn *= scaling;
  const size_t o = static_cast<size_t>(t) * 2 * half;
  cos_out[o + i] = cs;
  cos_out[o + half + i] = cs;
  sin_out[o + i] = sn;
  sin_out[o + half + i] = sn;
}

// x: [T, Hn, D] (row stride ldx elements between tokens), rotate-half convention:
// y[:half] = x1*c1 - x2*s1 ; y[half:] = x2*c2 + x1*s2.  `conj` applies the transpose
// (backward).  rot_dim <= D: dims beyond rot_dim are copied.
// W pairs per thread: 8 where the second half starts on a 16-byte boundary (rot_dim a multiple of 16), else 4 (heads of 72:
// the second half starts on an 8-byte one).  Bound by memory either way; a head of 72 through framework operations took
// eight passes in fp32.
template <int W>
__device__ __forceinline__ void load_w(const bf16* p, float (&v)[W]);
template <>
__device__ __forceinline__ void load_w<8>(const bf16* p, float (&v)[8]) { load8(p, v); }
template <>
__device__ __forceinline__ void load_w<4>(const bf16* p, float (&v)[4]) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template <int W>
__device__ __forceinline__ void store_w(bf16* p, const float (&v)[W]);
template <>
__device__ __forceinline__ void store_w<8>(bf16* p, const float (&v)[8]) { store8(p, v); }
template <>
__device__ __forceinline__ void store_w<4>(bf16* p, const float (&v)[4]) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
}

template <int W>
__global__ void rope_apply_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, const float* __restrict__ cosb,
                                  const float* __restrict__ sinb, int T, int Hn, int D, int rot_dim, long ldx,
                                  long ldy, int conj) {
  const int half = rot_dim / 2;
  const int per_head = half / W;  // vectors of W pairs
  const long total = static_cast<long>(T) * Hn * per_head;
  for (long idx = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long>(gridDim.x) * blockDim.x) {
    const int v = idx % per_head;
    const long th = idx / per_head;
    const int h = th % Hn;
    const long t = th / Hn;
    const bf16* xp = x + t * ldx + static_cast<long>(h) * D;
    bf16* yp = y + t * ldy + static_cast<long>(h) * D;
    float x1[W], x2[W], o1[W], o2[W];
    load_w<W>(xp + v * W, x1);
    load_w<W>(xp + half + v * W, x2);
    const float* c = cosb + t * rot_dim;
    const float* s = sinb + t * rot_dim;
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const float c1 = c[v * W + j], c2 = c[half + v * W + j];
      const float s1 = s[v * W + j], s2 = s[half + v * W + j];
      if (!conj) {
        o1[j] = x1[j] * c1 - x2[j] * s1;
        o2[j] = x2[j] * c2 + x1[j] * s2;
      } else {
        o1[j] = x1[j] * c1 + x2[j] * s2;
        o2[j] = x2[j] * c2 - x1[j] * s1;
      }
    }
    store_w<W>(yp + v * W, o1);
    store_w<W>(yp + half + v * W, o2);
  }
}

// ------------------------------------------------------------------ per-head RMSNorm + rotary embedding
// The q and k heads of a projection row [T, n_q + n_kv (+ ...), D] (row stride ldx): y = rope(rmsnorm(x) * w), the rotation over
// the whole head; D = 64 or 128.  D / 8 lanes share a head, eight columns each; the rotation's partner comes from the lane half
// a head away.  Sums run in the order of the separate norm kernels and every value is rounded where they store it, so that both
// forms give the same bits (a model of 28 layers amplifies any other rounding).  As separate passes a head was copied out of its
// strided row, normalised and rotated (six reads and writes of q and k); here it is read and written once.  Bound by memory.
__device__ __forceinline__ float group_sum(float v, int lanes) {
  for (int o = lanes >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void load_f8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <int D>
__global__ void __launch_bounds__(256) qk_norm_rope_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y,
                                                               const bf16* __restrict__ wq, const bf16* __restrict__ wk,
                                                               const float* __restrict__ cosb, const float* __restrict__ sinb,
                                                               float* __restrict__ rstd, long T, int n_q, int n_kv, long ldx,
                                                               long ldy, float eps) {
  constexpr int L = D / 8, HPW = 32 / L;   // lanes per head, heads per warp
  const int lane = threadIdx.x & 31, c = (lane % L) * 8, heads = n_q + n_kv;
  const bool lower = c < D / 2;
  const long total = T * heads;
  const bool narrow = fits32(total);
  const long warps = static_cast<long>(gridDim.x) * (blockDim.x >> 5);
  // every lane of a warp takes part in the shuffles: a group past the end computes on the last head and stores nothing
  for (long w0 = (static_cast<long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * HPW; w0 < total; w0 += warps * HPW) {
    const long idx = w0 + lane / L;
    const bool live = idx < total;
    const long at = live ? idx : total - 1;
    long t;
    int h;
    split_index(at, heads, narrow, t, h);
    float v[8], wv[8], cs[8], sn[8], o[8];
    load8(x + t * ldx + static_cast<long>(h) * D + c, v);
    load8((h < n_q ? wq : wk) + c, wv);
    load_f8(cosb + t * D + c, cs);
    load_f8(sinb + t * D + c, sn);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
    const float r = rsqrtf(group_sum(ss, L) / D + eps);
    if (live && lane % L == 0) rstd[at] = r;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float n = __bfloat162float(__float2bfloat16(v[j] * r * wv[j]));
      const float m = __shfl_xor_sync(0xffffffffu, n, L / 2);
      o[j] = lower ? n * cs[j] - m * sn[j] : n * cs[j] + m * sn[j];
    }
    if (live) store8(y + t * ldy + static_cast<long>(h) * D + c, o);
  }
}
// d [T, heads, D] (row stride ldd): gradient of y on entry, of x on exit; part [gridDim.x][2][D] partial weight gradients.
template <int D>
__global__ void __launch_bounds__(256) qk_norm_rope_bwd_kernel(bf16* d, const bf16* __restrict__ x, const bf16* __restrict__ wq,
                                                               const bf16* __restrict__ wk, const float* __restrict__ cosb,
                                                               const float* __restrict__ sinb, const float* __restrict__ rstd,
                                                               float* __restrict__ part, long T, int n_q, int n_kv, long ldx,
                                                               long ldd) {
  constexpr int L = D / 8, HPW = 32 / L;
  __shared__ float sw[2][D];
  const int lane = threadIdx.x & 31, l = lane % L, c = l * 8, heads = n_q + n_kv;
  const bool lower = c < D / 2;
  const int other = lower ? c + D / 2 : c - D / 2;
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) (&sw[0][0])[i] = 0.f;
  __syncthreads();
  float dw[2][8] = {};
  const long total = T * heads;
  const bool narrow = fits32(total);
  const long warps = static_cast<long>(gridDim.x) * (blockDim.x >> 5);
  for (long w0 = (static_cast<long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * HPW; w0 < total; w0 += warps * HPW) {
    const long idx = w0 + lane / L;
    const bool live = idx < total;
    const long at = live ? idx : total - 1;
    long t;
    int h;
    split_index(at, heads, narrow, t, h);
    bf16* dp = d + t * ldd + static_cast<long>(h) * D + c;
    float v[8], g[8], wv[8], cs[8], sn[8];
    load8(x + t * ldx + static_cast<long>(h) * D + c, v);
    load8(dp, g);
    const bool is_q = h < n_q;
    load8((is_q ? wq : wk) + c, wv);
    load_f8(cosb + t * D + c, cs);
    load_f8(sinb + t * D + other, sn);
    const float r = rstd[at];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      // transposed rotation, rounded where the separate form stores it
      const float m = __shfl_xor_sync(0xffffffffu, g[j], L / 2);
      const float dy = __bfloat162float(__float2bfloat16(lower ? g[j] * cs[j] + m * sn[j] : g[j] * cs[j] - m * sn[j]));
      v[j] *= r;
      // an index that depends on the head would put the sums into local memory
      const float s = live ? dy * v[j] : 0.f;
      dw[0][j] += is_q ? s : 0.f;
      dw[1][j] += is_q ? 0.f : s;
      g[j] = dy * wv[j];
      dot += g[j] * v[j];
    }
    dot = group_sum(dot, L) / D;
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = r * (g[j] - v[j] * dot);
    __syncwarp();   // a group past the end read the last head: it must have before that head is rewritten
    if (live) store8(dp, g);
  }
  // the groups of a warp in a fixed order, then the warps one after the other: the same sum on every run
#pragma unroll
  for (int k = 0; k < 2; ++k)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      for (int o = L; o < 32; o <<= 1) dw[k][j] += __shfl_xor_sync(0xffffffffu, dw[k][j], o);
  for (int wv = 0; wv < static_cast<int>(blockDim.x >> 5); ++wv) {
    if (static_cast<int>(threadIdx.x >> 5) == wv && lane < L) {
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 8; ++j) sw[k][c + j] += dw[k][j];
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < 2 * D; i += blockDim.x) part[static_cast<long>(blockIdx.x) * 2 * D + i] = (&sw[0][0])[i];
}

// ------------------------------------------------------------------ gated per-head RMSNorm (output of linear attention)
// y = bf16(rmsnorm(o) * w) * silu(z): o [T, heads, D] dense, z rows of contiguous heads at stride ldz (a column range of the
// projection), D = 8 L.  L lanes hold a head.  As framework operations the gate took seven passes over the rows, four of them in
// fp32, and the gate's columns were copied out first; bound by memory, each tensor is read or written once here.
template <int L>
__global__ void __launch_bounds__(256) gated_norm_fwd_kernel(const bf16* __restrict__ o, const bf16* __restrict__ z,
                                                             const bf16* __restrict__ w, bf16* __restrict__ y,
                                                             float* __restrict__ rstd_out, long rows, int heads, long ldz, float eps) {
  constexpr int D = 8 * L, HPW = 32 / L;
  const int lane = threadIdx.x & 31, c = (lane % L) * 8;
  const bool narrow = fits32(rows);
  const long warps = static_cast<long>(gridDim.x) * (blockDim.x >> 5);
  float wv[8];
  load8(w + c, wv);
  for (long w0 = (static_cast<long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * HPW; w0 < rows; w0 += warps * HPW) {
    const long r = w0 + lane / L;
    const bool live = r < rows;   // a group past the end takes part in the shuffles on the last row
    const long at = live ? r : rows - 1;
    long t;
    int h;
    split_index(at, heads, narrow, t, h);
    float v[8], zv[8], out[8];
    load8(o + at * D + c, v);
    load8(z + t * ldz + static_cast<long>(h) * D + c, zv);
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) ss += v[j] * v[j];
    const float rstd = rsqrtf(group_sum(ss, L) / D + eps);
#pragma unroll
    for (int j = 0; j < 8; ++j) out[j] = __bfloat162float(__float2bfloat16(v[j] * rstd * wv[j])) * (zv[j] / (1.f + expf(-zv[j])));
    if (live) {
      store8(y + at * D + c, out);
      if (lane % L == 0) rstd_out[at] = rstd;
    }
  }
}
template <int L>
__global__ void __launch_bounds__(256) gated_norm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ o,
                                                             const bf16* __restrict__ z, const bf16* __restrict__ w,
                                                             const float* __restrict__ rstd_in, bf16* __restrict__ d_o,
                                                             bf16* __restrict__ dz, float* __restrict__ part, long rows, int heads,
                                                             long ldz) {
  constexpr int D = 8 * L, HPW = 32 / L;
  __shared__ float sw[8][D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = (lane % L) * 8;
  const bool narrow = fits32(rows);
  const long warps = static_cast<long>(gridDim.x) * 8;
  float wv[8], dw[8];
  load8(w + c, wv);
#pragma unroll
  for (int j = 0; j < 8; ++j) dw[j] = 0.f;
  for (long w0 = (static_cast<long>(blockIdx.x) * 8 + warp) * HPW; w0 < rows; w0 += warps * HPW) {
    const long r = w0 + lane / L;
    const bool live = r < rows;
    const long at = live ? r : rows - 1;
    long t;
    int h;
    split_index(at, heads, narrow, t, h);
    float g[8], v[8], zv[8], gz[8];
    load8(dy + at * D + c, g);
    load8(o + at * D + c, v);
    load8(z + t * ldz + static_cast<long>(h) * D + c, zv);
    const float rstd = rstd_in[at];
    float dot = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sig = 1.f / (1.f + expf(-zv[j])), si = zv[j] * sig;
      v[j] *= rstd;
      const float n = __bfloat162float(__float2bfloat16(v[j] * wv[j]));
      gz[j] = g[j] * n * (sig * (1.f + zv[j] * (1.f - sig)));
      const float dn = __bfloat162float(__float2bfloat16(g[j] * si));   // a bf16 tensor in the separate form
      if (live) dw[j] += dn * v[j];
      g[j] = dn * wv[j];
      dot += g[j] * v[j];
    }
    dot = group_sum(dot, L) / D;
#pragma unroll
    for (int j = 0; j < 8; ++j) g[j] = rstd * (g[j] - v[j] * dot);
    if (live) {
      store8(d_o + at * D + c, g);
      store8(dz + at * D + c, gz);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
    for (int k = L; k < 32; k <<= 1) dw[j] += __shfl_xor_sync(0xffffffffu, dw[j], k);
  if (lane < L) {
#pragma unroll
    for (int j = 0; j < 8; ++j) sw[warp][c + j] = dw[j];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < D; i += 256) {
    float s = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) s += sw[q][i];
    part[static_cast<long>(blockIdx.x) * D + i] = s;
  }
}

// ------------------------------------------------------------------ SwiGLU
__global__ void swiglu_fwd_kernel(const bf16* __restrict__ g, const bf16* __restrict__ u, bf16* __restrict__ h,
                                  long n8) {
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n8;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    float gv[8], uv[8], o[8];
    load8(g + i * 8, gv);
    load8(u + i * 8, uv);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = gv[j] / (1.f + __expf(-gv[j])) * uv[j];
    store8(h + i * 8, o);
  }
}
// dg, du may alias g, u (in place).
__global__ void swiglu_bwd_kernel(const bf16* __restrict__ dh, const bf16* g, const bf16* u, bf16* dg, bf16* du,
                                  long n8) {
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n8;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    float dv[8], gv[8], uv[8], og[8], ou[8];
    load8(dh + i * 8, dv);
    load8(g + i * 8, gv);
    load8(u + i * 8, uv);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float sig = 1.f / (1.f + __expf(-gv[j]));
      const float silu = gv[j] * sig;
      ou[j] = dv[j] * silu;
      og[j] = dv[j] * uv[j] * (sig + silu * (1.f - sig));
    }
    store8(dg + i * 8, og);
    store8(du + i * 8, ou);
  }
}

// ------------------------------------------------------------------ optimizers on flat buffers
// AdamW with fp32 master weights and moments; gradient bf16 or fp32.  `gscale` (device
// scalar, may be null) multiplies the gradient (clip coefficient); `skip` (device int,
// may be null) suppresses the whole update when non-zero (non-finite gradient norm).
template <typename GT>
__global__ void adamw_kernel(float* __restrict__ p32, bf16* __restrict__ p16, float* __restrict__ m,
                             float* __restrict__ v, const GT* __restrict__ g, long n, float lr, float beta1,
                             float beta2, float eps, float wd, float bc1, float bc2, const float* gscale,
                             const int* skip) {
  if (skip != nullptr && *skip) return;
  const float gs = gscale != nullptr ? *gscale : 1.f;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float gi = static_cast<float>(g[i]) * gs;
    float pi = p32[i];
    const float mi = beta1 * m[i] + (1.f - beta1) * gi;
    const float vi = beta2 * v[i] + (1.f - beta2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    pi *= (1.f - lr * wd);
    pi -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p32[i] = pi;
    if (p16 != nullptr) p16[i] = __float2bfloat16(pi);
  }
}

// Muon step 1: momentum and the Newton-Schulz input.
//   mom = beta*mom + (1-beta)*g ; u = nesterov ? g + beta*(mom - g) : mom ; out = bf16(u)
// plus the sum of squares of u into sumsq[0] (one atomic per CTA) for the Frobenius norm.
template <typename GT>
__global__ void muon_momentum_kernel(float* __restrict__ mom, const GT* __restrict__ g, bf16* __restrict__ out,
                                     float* __restrict__ sumsq, long n, float beta, int nesterov,
                                     const float* gscale) {
  __shared__ float red[32];
  const float gs = gscale != nullptr ? *gscale : 1.f;
  float acc = 0.f;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float gi = static_cast<float>(g[i]) * gs;
    const float mi = beta * mom[i] + (1.f - beta) * gi;
    mom[i] = mi;
    const float u = nesterov ? gi + beta * (mi - gi) : mi;
    out[i] = __float2bfloat16(u);
    acc += u * u;
  }
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) atomicAdd(sumsq, acc);
}
// x *= 1 / (sqrt(sumsq) + eps)   (bf16 in place)
__global__ void scale_by_norm_kernel(bf16* __restrict__ x, const float* __restrict__ sumsq, long n, float eps) {
  const float s = 1.f / (sqrtf(*sumsq) + eps);
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x)
    x[i] = __float2bfloat16(__bfloat162float(x[i]) * s);
}
// Muon step 3: p = p*(1 - lr*wd) - lr*scale*o ; bf16 copy refreshed.
__global__ void muon_update_kernel(float* __restrict__ p32, bf16* __restrict__ p16, const bf16* __restrict__ o,
                                   long n, float lr, float wd, float scale, const int* skip) {
  if (skip != nullptr && *skip) return;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    float pi = p32[i] * (1.f - lr * wd) - lr * scale * __bfloat162float(o[i]);
    p32[i] = pi;
    if (p16 != nullptr) p16[i] = __float2bfloat16(pi);
  }
}

// ema = decay*ema + (1-decay)*p
template <typename PT>
__global__ void ema_kernel(float* __restrict__ ema, const PT* __restrict__ p, long n, float decay) {
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x)
    ema[i] = decay * ema[i] + (1.f - decay) * static_cast<float>(p[i]);
}

// ---- 16-byte versions of the optimizer passes ---------------------------------------------------------------
// The passes above move 2 or 4 bytes per thread and iteration, which keeps too few bytes in flight to fill HBM
// (1.3 - 3.5 TB/s measured).  These take four elements per thread and iteration (float4 / 4 x bf16); the launchers use
// them when every pointer is 16-byte aligned (8 for the bf16 arrays) and hand the last n % 4 elements to the scalar
// kernels.  Element-wise results are bit-identical to the scalar kernels; the sums of squares add in another order.
struct alignas(8) bf16x4 {
  uint32_t lo, hi;
};
__device__ __forceinline__ bf16x4 to_bf16x4(float a, float b, float c, float d) {
  bf16x4 r;
  r.lo = pack_bf16x2(a, b);
  r.hi = pack_bf16x2(c, d);
  return r;
}

// four gradient elements of either type
__device__ __forceinline__ float4 grad4(const float4& g) { return g; }
__device__ __forceinline__ float4 grad4(const bf16x4& g) {
  const float2 a = unpack_bf16x2(g.lo), b = unpack_bf16x2(g.hi);
  return make_float4(a.x, a.y, b.x, b.y);
}

template <typename G4>
__global__ void adamw_vec_kernel(float4* __restrict__ p32, bf16x4* __restrict__ p16, float4* __restrict__ m,
                                 float4* __restrict__ v, const G4* __restrict__ g, long nv, float lr, float beta1,
                                 float beta2, float eps, float wd, float bc1, float bc2, const float* gscale,
                                 const int* skip) {
  if (skip != nullptr && *skip) return;
  const float gs = gscale != nullptr ? *gscale : 1.f;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nv;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float4 g4 = grad4(g[i]);
    float4 p4 = p32[i], m4 = m[i], v4 = v[i];
    const float gi[4] = {g4.x * gs, g4.y * gs, g4.z * gs, g4.w * gs};
    float pi[4] = {p4.x, p4.y, p4.z, p4.w}, mi[4] = {m4.x, m4.y, m4.z, m4.w}, vi[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      mi[e] = beta1 * mi[e] + (1.f - beta1) * gi[e];
      vi[e] = beta2 * vi[e] + (1.f - beta2) * gi[e] * gi[e];
      pi[e] *= (1.f - lr * wd);
      pi[e] -= lr * (mi[e] / bc1) / (sqrtf(vi[e] / bc2) + eps);
    }
    m[i] = make_float4(mi[0], mi[1], mi[2], mi[3]);
    v[i] = make_float4(vi[0], vi[1], vi[2], vi[3]);
    p32[i] = make_float4(pi[0], pi[1], pi[2], pi[3]);
    if (p16 != nullptr) p16[i] = to_bf16x4(pi[0], pi[1], pi[2], pi[3]);
  }
}

template <typename G4>
__global__ void muon_momentum_vec_kernel(float4* __restrict__ mom, const G4* __restrict__ g, bf16x4* __restrict__ out,
                                         float* __restrict__ sumsq, long nv, float beta, int nesterov,
                                         const float* gscale) {
  __shared__ float red[32];
  const float gs = gscale != nullptr ? *gscale : 1.f;
  float acc = 0.f;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nv;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float4 g4 = grad4(g[i]);
    const float4 m4 = mom[i];
    const float gi[4] = {g4.x * gs, g4.y * gs, g4.z * gs, g4.w * gs};
    float mi[4] = {m4.x, m4.y, m4.z, m4.w}, u[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      mi[e] = beta * mi[e] + (1.f - beta) * gi[e];
      u[e] = nesterov ? gi[e] + beta * (mi[e] - gi[e]) : mi[e];
      acc += u[e] * u[e];
    }
    mom[i] = make_float4(mi[0], mi[1], mi[2], mi[3]);
    out[i] = to_bf16x4(u[0], u[1], u[2], u[3]);
  }
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) atomicAdd(sumsq, acc);
}

__global__ void scale_by_norm_vec_kernel(uint4* __restrict__ x, const float* __restrict__ sumsq, long nv8, float eps) {
  const float s = 1.f / (sqrtf(*sumsq) + eps);
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nv8;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    uint4 w = x[i];
    float2 a = unpack_bf16x2(w.x), b = unpack_bf16x2(w.y), c = unpack_bf16x2(w.z), d = unpack_bf16x2(w.w);
    // the same rounding as the scalar kernel: bf16(float(x) * s)
    w.x = pack_bf16x2(a.x * s, a.y * s);
    w.y = pack_bf16x2(b.x * s, b.y * s);
    w.z = pack_bf16x2(c.x * s, c.y * s);
    w.w = pack_bf16x2(d.x * s, d.y * s);
    x[i] = w;
  }
}

__global__ void muon_update_vec_kernel(float4* __restrict__ p32, bf16x4* __restrict__ p16, const bf16x4* __restrict__ o,
                                       long nv, float lr, float wd, float scale, const int* skip) {
  if (skip != nullptr && *skip) return;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < nv;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float4 p4 = p32[i];
    const bf16x4 o4 = o[i];
    const float2 oa = unpack_bf16x2(o4.lo), ob = unpack_bf16x2(o4.hi);
    const float r0 = p4.x * (1.f - lr * wd) - lr * scale * oa.x;
    const float r1 = p4.y * (1.f - lr * wd) - lr * scale * oa.y;
    const float r2 = p4.z * (1.f - lr * wd) - lr * scale * ob.x;
    const float r3 = p4.w * (1.f - lr * wd) - lr * scale * ob.y;
    p32[i] = make_float4(r0, r1, r2, r3);
    if (p16 != nullptr) p16[i] = to_bf16x4(r0, r1, r2, r3);
  }
}

__global__ void sumsq_part_vec_kernel(const float4* __restrict__ g, float* __restrict__ part, long nv, const float* tail,
                                      int n_tail) {
  __shared__ float red[32];
  float acc = 0.f;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x;
  long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  // four independent 16-byte loads per thread and iteration: the grid is capped at the size of the partials scratch
  for (; i + 3 * stride < nv; i += 4 * stride) {
    const float4 a = g[i], b = g[i + stride], c = g[i + 2 * stride], d = g[i + 3 * stride];
    acc += (a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w) + (b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w) +
           (c.x * c.x + c.y * c.y + c.z * c.z + c.w * c.w) + (d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w);
  }
  for (; i < nv; i += stride) {
    const float4 v = g[i];
    acc += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
  }
  if (blockIdx.x == 0 && threadIdx.x < n_tail) acc += tail[threadIdx.x] * tail[threadIdx.x];
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

__device__ __forceinline__ float sq8(const uint4& w) {
  const float2 a = unpack_bf16x2(w.x), b = unpack_bf16x2(w.y), c = unpack_bf16x2(w.z), d = unpack_bf16x2(w.w);
  return (a.x * a.x + a.y * a.y + b.x * b.x + b.y * b.y) + (c.x * c.x + c.y * c.y + d.x * d.x + d.y * d.y);
}
// The same over bf16, eight elements a load and eight loads in flight: two CTAs per SM (the partials) need 64 KB per SM under
// way to reach HBM's rate.
__global__ void sumsq_part_bf16_kernel(const uint4* __restrict__ g, float* __restrict__ part, long nv, const bf16* tail, int n_tail) {
  __shared__ float red[32];
  float acc = 0.f;
  const long stride = static_cast<long>(gridDim.x) * blockDim.x;
  long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x;
  for (; i + 7 * stride < nv; i += 8 * stride) {
    uint4 w[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) w[j] = g[i + j * stride];
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += sq8(w[j]);
    acc += s;
  }
  for (; i < nv; i += stride) acc += sq8(g[i]);
  if (blockIdx.x == 0 && static_cast<int>(threadIdx.x) < n_tail) {
    const float t = __bfloat162float(tail[threadIdx.x]);
    acc += t * t;
  }
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}

// LMMS_B200_SCALAR_OPTIM=1 keeps the scalar passes (the A/B of profiles/optimizer_passes_microbench.md)
static inline bool aligned_to(const void* p, uintptr_t a) {
  static const bool scalar_only = [] {
    const char* e = getenv("LMMS_B200_SCALAR_OPTIM");
    return e != nullptr && e[0] == '1';
  }();
  return !scalar_only && (p == nullptr || (reinterpret_cast<uintptr_t>(p) % a) == 0);
}

// Deterministic two-stage sum of squares: part[blockIdx.x] then a single-CTA finish.
template <typename GT>
__global__ void sumsq_part_kernel(const GT* __restrict__ g, float* __restrict__ part, long n) {
  __shared__ float red[32];
  float acc = 0.f;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    const float gi = static_cast<float>(g[i]);
    acc += gi * gi;
  }
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) part[blockIdx.x] = acc;
}
// out[0] (+)= sum(part)
__global__ void sumsq_finish_kernel(const float* __restrict__ part, float* __restrict__ out, int parts,
                                    int accumulate) {
  __shared__ float red[32];
  float acc = 0.f;
  for (int i = threadIdx.x; i < parts; i += blockDim.x) acc += part[i];
  acc = block_sum<256>(acc, red);
  if (threadIdx.x == 0) out[0] = accumulate ? out[0] + acc : acc;
}
// From the global sum of squares: norm, clip coefficient min(1, max_norm/(norm+1e-6)),
// and a skip flag when the norm is not finite or a kernel of this device has raised the status
// word (a bounded wait that ran out: the gradients of this step may be incomplete).  No host
// round trip.
__global__ void clip_coef_kernel(const float* __restrict__ sumsq, float* __restrict__ norm_out,
                                 float* __restrict__ coef_out, int* __restrict__ skip_out, float max_norm,
                                 const int* __restrict__ status) {
  const float norm = sqrtf(*sumsq);
  *norm_out = norm;
  const bool finite = isfinite(norm);
  const bool faulted = status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
  *skip_out = (finite && !faulted) ? 0 : 1;
  float c = 1.f;
  if (max_norm > 0.f && finite) c = fminf(1.f, max_norm / (norm + 1e-6f));
  *coef_out = c;
}
template <typename GT>
__global__ void scale_kernel(GT* __restrict__ g, long n, const float* __restrict__ coef) {
  const float c = *coef;
  if (c == 1.f) return;
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<long>(gridDim.x) * blockDim.x)
    g[i] = static_cast<GT>(static_cast<float>(g[i]) * c);
}

// ------------------------------------------------------------------ packed-sequence index kernels
// out[i, :] = src[idx[i], :]  (idx < 0 writes zeros) and the scatter inverse (optionally adding).
__global__ void gather_rows_kernel(const bf16* __restrict__ src, const int64_t* __restrict__ idx,
                                   bf16* __restrict__ out, long n_out, int H, long n_src, int* status) {
  const int vec = H / 8;
  const long total = n_out * vec;
  const bool narrow = fits32(total);
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    long r;
    int c;
    split_index(i, vec, narrow, r, c);
    c *= 8;
    const int64_t s = idx[r];
    bf16x8 v;
    v.w[0] = v.w[1] = v.w[2] = v.w[3] = 0u;
    if (s >= 0 && index_in_bounds(s, n_src, status)) v = *reinterpret_cast<const bf16x8*>(src + s * H + c);
    *reinterpret_cast<bf16x8*>(out + r * H + c) = v;
  }
}
__global__ void scatter_rows_kernel(const bf16* __restrict__ src, const int64_t* __restrict__ idx,
                                    bf16* __restrict__ out, long n_src, int H, int add, long n_out, int* status) {
  const int vec = H / 8;
  const long total = n_src * vec;
  const bool narrow = fits32(total);
  for (long i = blockIdx.x * static_cast<long>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<long>(gridDim.x) * blockDim.x) {
    long r;
    int c;
    split_index(i, vec, narrow, r, c);
    c *= 8;
    const int64_t d = idx[r];
    if (d < 0 || !index_in_bounds(d, n_out, status)) continue;
    float v[8];
    load8(src + r * H + c, v);
    if (add) {
      float o[8];
      load8(out + d * H + c, o);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] += o[j];
    }
    store8(out + d * H + c, v);
  }
}

// ------------------------------------------------------------------ cross-entropy passes
// After the logits GEMM with the statistics epilogue: combine the per-tile partials into
// lse, pick the target logit, emit per-row loss (0 for ignored rows).
__global__ void ce_finalize_kernel(const float2* __restrict__ stats, const bf16* __restrict__ logits,
                                   const int64_t* __restrict__ labels, float* __restrict__ lse_out,
                                   float* __restrict__ loss_out, int rows, int n_tiles, long ld, int V,
                                   int ignore_index) {
  const int lane = threadIdx.x & 31;
  const int wpb = blockDim.x >> 5;
  for (int row = blockIdx.x * wpb + (threadIdx.x >> 5); row < rows; row += gridDim.x * wpb) {
    float mx = -INFINITY;
    for (int i = lane; i < n_tiles; i += 32) mx = fmaxf(mx, stats[static_cast<size_t>(row) * n_tiles + i].x);
    mx = warp_max(mx);
    float s = 0.f;
    for (int i = lane; i < n_tiles; i += 32) {
      const float2 st = stats[static_cast<size_t>(row) * n_tiles + i];
      if (st.x > -INFINITY) s += st.y * __expf(st.x - mx);
    }
    s = warp_sum(s);
    if (lane == 0) {
      const float lse = mx + logf(s);
      lse_out[row] = lse;
      const int64_t y = labels[row];
      float l = 0.f;
      if (y != ignore_index && y >= 0 && y < V) l = lse - __bfloat162float(logits[static_cast<size_t>(row) * ld + y]);
      loss_out[row] = l;
    }
  }
}
// In place: logits[r, c] <- gscale[0]*row_w * (exp(logits - lse) - [c == label]); ignored rows -> 0.
__global__ void ce_dlogits_kernel(bf16* __restrict__ logits, const float* __restrict__ lse,
                                  const int64_t* __restrict__ labels, const float* __restrict__ gscale, int rows,
                                  long ld, int V, int ignore_index) {
  const int vec = V / 8;
  const float gs = *gscale;
  for (int row = blockIdx.y; row < rows; row += gridDim.y) {
    const int64_t y = labels[row];
    const bool ign = (y == ignore_index);
    const float l = lse[row];
    bf16* base = logits + static_cast<size_t>(row) * ld;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < vec; i += gridDim.x * blockDim.x) {
      float v[8];
      if (ign) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.f;
      } else {
        load8(base + i * 8, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float pr = __expf(v[j] - l);
          if (i * 8 + j == y) pr -= 1.f;
          v[j] = pr * gs;
        }
      }
      store8(base + i * 8, v);
    }
  }
}

static int g_sms = 0;
static int num_sms() {
  if (g_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev);
  }
  return g_sms;
}
static int grid_for(long work_items, int threads, int per_sm = 8) {
  long blocks = (work_items + threads - 1) / threads;
  long cap = static_cast<long>(num_sms()) * per_sm;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return static_cast<int>(blocks);
}

}  // namespace b200

using namespace b200;

#define CHECK_LAUNCH() (cudaGetLastError() == cudaSuccess ? 0 : -4)

extern "C" {

int b200_num_partials() { return num_sms() * 2; }

// rows x H bf16.  ln = 0: RMSNorm, 1: LayerNorm (b may be null).  res/res_out may be null.
int b200_norm_fwd(const void* x, const void* res, const void* w, const void* b, void* y, void* res_out, void* rstd,
                  void* mean, int rows, int H, float eps, float w_offset, int ln, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (H % 8) return -10;
  if (H <= 512 && !ln && res == nullptr) {
    int blocks = grid_for(static_cast<long>(rows) * 32, 256, 8);
    norm_fwd_warp_kernel<<<blocks, 256, 0, st>>>((const bf16*)x, (const bf16*)w, (bf16*)y, (float*)rstd, rows, H, eps,
                                                 w_offset);
    return CHECK_LAUNCH();
  }
  int blocks = rows < num_sms() * 8 ? rows : num_sms() * 8;
#define NORM_FWD(T, V)                                                                                              \
  norm_fwd_kernel<T, V><<<blocks, T, 0, st>>>((const bf16*)x, (const bf16*)res, (const bf16*)w, (const bf16*)b,     \
                                              (bf16*)y, (bf16*)res_out, (float*)rstd, (float*)mean, rows, H, eps, \
                                              w_offset, ln)
  if (H <= 1024) NORM_FWD(128, 1);
  else if (H <= 2048) NORM_FWD(256, 1);
  else if (H <= 4096) NORM_FWD(256, 2);
  else if (H <= 8192) NORM_FWD(512, 2);
  else if (H <= 16384) NORM_FWD(512, 4);
  else return -11;
#undef NORM_FWD
  return CHECK_LAUNCH();
}

// dw_part / db_part: fp32 [b200_num_partials(), H] scratch.  dw/db fp32 [H] (accumulate flag).
int b200_norm_bwd(const void* dy, const void* x, const void* w, const void* rstd, const void* mean,
                  const void* dres_in, void* dx, void* dw_part, void* db_part, void* dw, void* db, int rows, int H,
                  float w_offset, int ln, int accumulate, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (H % 8) return -10;
  int parts;
  if (H <= 512 && !ln && dres_in == nullptr) {
    if (H == 64 || H == 128 || H == 256) {
      const int lpr = H / 8, rows_per_block = 16 * (32 / lpr);
      long want = (static_cast<long>(rows) + rows_per_block - 1) / rows_per_block;
      parts = static_cast<int>(want < num_sms() * 2 ? want : num_sms() * 2);  // one partials row per block
      if (parts < 1) parts = 1;
      if (H == 64)
        norm_bwd_narrow_kernel<8><<<parts, 512, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd,
                                                         (bf16*)dx, (float*)dw_part, rows, w_offset);
      else if (H == 128)
        norm_bwd_narrow_kernel<16><<<parts, 512, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd,
                                                          (bf16*)dx, (float*)dw_part, rows, w_offset);
      else
        norm_bwd_narrow_kernel<32><<<parts, 512, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd,
                                                          (bf16*)dx, (float*)dw_part, rows, w_offset);
      if (cudaGetLastError() != cudaSuccess) return -4;
      colsum((const float*)dw_part, (float*)dw, parts, H, accumulate, st);
      return CHECK_LAUNCH();
    }
    int blocks = num_sms() * 2 / 8;
    if (blocks < 1) blocks = 1;
    parts = blocks * 8;
    norm_bwd_warp_kernel<<<blocks, 256, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd,
                                                 (bf16*)dx, (float*)dw_part, rows, H, w_offset);
  } else if (H <= 2048 && !(ln && dres_in != nullptr)) {  // a LayerNorm with a residual's gradient has no caller among the layers
    // one row of partials per CTA; above 1024 columns the registers of a row leave one CTA per SM
    // A tile holds a row's registers, and what the row does not fill is idle.  22000 rows, RMS / LayerNorm, us: 1152 and 1280
    // columns (both vision towers) 55 / 70 on a tile of 1280, 63 / 81 on one of 2048; 1536 and 1792 columns, which no
    // configuration here has, take the tile of 2048 with 68 / 86 and 74 / 93 (tiles of their own: 63 / 80 and 72 / 89).
    parts = H <= 1024 ? num_sms() * 2 : num_sms();
    if (parts > (rows + 7) / 8) parts = (rows + 7) / 8;
#define NORM_BWD(V, L, R)                                                                                                \
  norm_bwd_rows_kernel<V, L, R><<<parts, 256, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd, \
                                                       (const float*)mean, (const bf16*)dres_in, (bf16*)dx, (float*)dw_part, \
                                                       (float*)db_part, rows, H, w_offset)
#define NORM_BWD_V(V)                       \
  do {                                      \
    if (ln) NORM_BWD(V, true, false);       \
    else if (dres_in) NORM_BWD(V, false, true);   \
    else NORM_BWD(V, false, false);         \
  } while (0)
    if (H <= 512) NORM_BWD_V(2);
    else if (H <= 1024) NORM_BWD_V(4);
    else if (H <= 1280) NORM_BWD_V(5);
    else NORM_BWD_V(8);
#undef NORM_BWD_V
#undef NORM_BWD
  } else {
    parts = num_sms() * 2;
    if (parts > rows) parts = rows;
#define NORM_BWD(T, V)                                                                                            \
  norm_bwd_kernel<T, V><<<parts, T, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd, \
                                             (const float*)mean, (const bf16*)dres_in, (bf16*)dx, (float*)dw_part, \
                                             (float*)db_part, rows, H, w_offset, ln)
    if (H <= 4096) NORM_BWD(256, 2);
    else if (H <= 8192) NORM_BWD(512, 2);
    else if (H <= 16384) NORM_BWD(512, 4);
    else return -11;
#undef NORM_BWD
  }
  if (cudaGetLastError() != cudaSuccess) return -4;
  colsum((const float*)dw_part, (float*)dw, parts, H, accumulate, st);
  if (db != nullptr && db_part != nullptr)
    colsum((const float*)db_part, (float*)db, parts, H, accumulate, st);
  return CHECK_LAUNCH();
}

// Rows of partials [this, N] fp32 that b200_colsum_bf16 needs.
int b200_colsum_parts(int rows, int N) {
  const int cols = (N + 255) / 256;
  int parts = num_sms() * 4 / (cols > 0 ? cols : 1);
  const int most = (rows + 31) / 32;   // at least four rows a warp
  if (parts > most) parts = most;
  return parts < 1 ? 1 : parts;
}
// out [N] bf16 = column sums of x [rows, N] bf16, rows ld elements apart (a multiple of 8, at least N rounded up to 8), 16-byte aligned.
int b200_colsum_bf16(const void* x, long ld, void* part, void* out, int rows, int N, int parts, cudaStream_t st) {
  if (N <= 0) return 0;
  if (ld % 8 || ld < (N + 7) / 8 * 8 || parts < 1 || parts > 65535) return -10;
  colsum_bf16_kernel<<<dim3((N + 255) / 256, parts), 256, 0, st>>>((const bf16*)x, ld, (float*)part, rows, N);
  colsum_bf16_finish_kernel<<<(N + 31) / 32, 1024, 0, st>>>((const float*)part, (bf16*)out, parts, N);
  return CHECK_LAUNCH();
}

int b200_rope_table(const void* pos, const void* inv_freq, void* cos_out, void* sin_out, int T, int half, int mode,
                    int s0, int s1, int s2, float scaling, cudaStream_t st) {
  long n = static_cast<long>(T) * half;
  if (n <= 0) return 0;
  rope_table_kernel<<<(n + 255) / 256, 256, 0, st>>>((const int64_t*)pos, (const float*)inv_freq, (float*)cos_out,
                                                     (float*)sin_out, T, half, mode, s0, s1, s2, scaling);
  return CHECK_LAUNCH();
}

int b200_rope_apply(const void* x, void* y, const void* cosb, const void* sinb, int T, int Hn, int D, int rot_dim,
                    long ldx, long ldy, int conj, cudaStream_t st) {
  if (T <= 0) return 0;
  if (rot_dim % 8 || D % 8 || ldx % 8 || ldy % 8) return -10;
  if (rot_dim % 16 == 0) {
    const long total = static_cast<long>(T) * Hn * (rot_dim / 16);
    rope_apply_kernel<8><<<grid_for(total, 256), 256, 0, st>>>((const bf16*)x, (bf16*)y, (const float*)cosb, (const float*)sinb, T, Hn, D,
                                                               rot_dim, ldx, ldy, conj);
  } else {
    const long total = static_cast<long>(T) * Hn * (rot_dim / 8);
    rope_apply_kernel<4><<<grid_for(total, 256), 256, 0, st>>>((const bf16*)x, (bf16*)y, (const float*)cosb, (const float*)sinb, T, Hn, D,
                                                               rot_dim, ldx, ldy, conj);
  }
  return CHECK_LAUNCH();
}

// Partial weight gradients that b200_qk_norm_rope_bwd writes: part [this][2][D] fp32.
int b200_qk_norm_rope_parts() { return num_sms() * 3; }  // as many CTAs as its registers keep resident

// q and k heads of rows x [T, >= (n_q + n_kv) * D] into y; D 64 or 128, rows on 16-byte boundaries, rstd [T, n_q + n_kv].
int b200_qk_norm_rope_fwd(const void* x, void* y, const void* wq, const void* wk, const void* cosb, const void* sinb, void* rstd,
                          long T, int n_q, int n_kv, int D, long ldx, long ldy, float eps, cudaStream_t st) {
  if (T <= 0) return 0;
  if ((D != 64 && D != 128) || ldx % 8 || ldy % 8 || n_q + n_kv <= 0) return -10;
  const int blocks = grid_for(T * (n_q + n_kv) * (D / 8), 256);
  if (D == 128)
    qk_norm_rope_fwd_kernel<128><<<blocks, 256, 0, st>>>((const bf16*)x, (bf16*)y, (const bf16*)wq, (const bf16*)wk, (const float*)cosb,
                                                         (const float*)sinb, (float*)rstd, T, n_q, n_kv, ldx, ldy, eps);
  else
    qk_norm_rope_fwd_kernel<64><<<blocks, 256, 0, st>>>((const bf16*)x, (bf16*)y, (const bf16*)wq, (const bf16*)wk, (const float*)cosb,
                                                        (const float*)sinb, (float*)rstd, T, n_q, n_kv, ldx, ldy, eps);
  return CHECK_LAUNCH();
}
int b200_qk_norm_rope_bwd(void* d, const void* x, const void* wq, const void* wk, const void* cosb, const void* sinb, const void* rstd,
                          void* part, long T, int n_q, int n_kv, int D, long ldx, long ldd, cudaStream_t st) {
  if ((D != 64 && D != 128) || ldx % 8 || ldd % 8 || n_q + n_kv <= 0 || T <= 0) return -10;
  const int blocks = b200_qk_norm_rope_parts();
  if (D == 128)
    qk_norm_rope_bwd_kernel<128><<<blocks, 256, 0, st>>>((bf16*)d, (const bf16*)x, (const bf16*)wq, (const bf16*)wk, (const float*)cosb,
                                                         (const float*)sinb, (const float*)rstd, (float*)part, T, n_q, n_kv, ldx, ldd);
  else
    qk_norm_rope_bwd_kernel<64><<<blocks, 256, 0, st>>>((bf16*)d, (const bf16*)x, (const bf16*)wq, (const bf16*)wk, (const float*)cosb,
                                                        (const float*)sinb, (const float*)rstd, (float*)part, T, n_q, n_kv, ldx, ldd);
  return CHECK_LAUNCH();
}

// o, y [rows, D] dense with rows = T * heads, z [T, >= heads * D] at row stride ldz (a multiple of 8), w [D]; D = 64, 128 or 256.
int b200_gated_norm_fwd(const void* o, const void* z, const void* w, void* y, void* rstd, long rows, int heads, int D, long ldz, float eps,
                        cudaStream_t st) {
  if (rows <= 0) return 0;
  if (heads <= 0 || ldz % 8) return -10;
  const int blocks = grid_for(rows * (D / 8), 256);
#define GATED(L) gated_norm_fwd_kernel<L><<<blocks, 256, 0, st>>>((const bf16*)o, (const bf16*)z, (const bf16*)w, (bf16*)y, (float*)rstd, rows, heads, ldz, eps)
  if (D == 64) GATED(8);
  else if (D == 128) GATED(16);
  else if (D == 256) GATED(32);
  else return -11;
#undef GATED
  return CHECK_LAUNCH();
}
// Rows of partial weight gradients [this, D] fp32 that the backward pass writes.
int b200_gated_norm_parts() { return num_sms() * 4; }
int b200_gated_norm_bwd(const void* dy, const void* o, const void* z, const void* w, const void* rstd, void* d_o, void* dz, void* part,
                        long rows, int heads, int D, long ldz, cudaStream_t st) {
  if (heads <= 0 || ldz % 8 || rows <= 0) return -10;
  const int blocks = b200_gated_norm_parts();
#define GATED(L) gated_norm_bwd_kernel<L><<<blocks, 256, 0, st>>>((const bf16*)dy, (const bf16*)o, (const bf16*)z, (const bf16*)w, (const float*)rstd, (bf16*)d_o, (bf16*)dz, (float*)part, rows, heads, ldz)
  if (D == 64) GATED(8);
  else if (D == 128) GATED(16);
  else if (D == 256) GATED(32);
  else return -11;
#undef GATED
  return CHECK_LAUNCH();
}

int b200_swiglu_fwd(const void* g, const void* u, void* h, long n, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  swiglu_fwd_kernel<<<grid_for(n / 8, 256), 256, 0, st>>>((const bf16*)g, (const bf16*)u, (bf16*)h, n / 8);
  return CHECK_LAUNCH();
}
int b200_swiglu_bwd(const void* dh, const void* g, const void* u, void* dg, void* du, long n, cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 8) return -10;
  swiglu_bwd_kernel<<<grid_for(n / 8, 256), 256, 0, st>>>((const bf16*)dh, (const bf16*)g, (const bf16*)u, (bf16*)dg,
                                                          (bf16*)du, n / 8);
  return CHECK_LAUNCH();
}

int b200_adamw(void* p32, void* p16, void* m, void* v, const void* g, int g_is_fp32, long n, float lr, float beta1,
               float beta2, float eps, float wd, float bc1, float bc2, const void* gscale, const void* skip,
               cudaStream_t st) {
  if (n <= 0) return 0;
  if (n >= 4 && aligned_to(p32, 16) && aligned_to(p16, 8) && aligned_to(m, 16) && aligned_to(v, 16) && aligned_to(g, g_is_fp32 ? 16 : 8)) {
    const long nv = n / 4, done = nv * 4;
    bf16* tail16 = p16 ? (bf16*)p16 + done : nullptr;
    if (g_is_fp32) {
      adamw_vec_kernel<<<grid_for(nv, 256), 256, 0, st>>>((float4*)p32, (bf16x4*)p16, (float4*)m, (float4*)v, (const float4*)g, nv, lr,
                                                          beta1, beta2, eps, wd, bc1, bc2, (const float*)gscale, (const int*)skip);
      if (done < n)
        adamw_kernel<float><<<1, 32, 0, st>>>((float*)p32 + done, tail16, (float*)m + done, (float*)v + done, (const float*)g + done,
                                              n - done, lr, beta1, beta2, eps, wd, bc1, bc2, (const float*)gscale, (const int*)skip);
    } else {
      adamw_vec_kernel<<<grid_for(nv, 256), 256, 0, st>>>((float4*)p32, (bf16x4*)p16, (float4*)m, (float4*)v, (const bf16x4*)g, nv, lr,
                                                          beta1, beta2, eps, wd, bc1, bc2, (const float*)gscale, (const int*)skip);
      if (done < n)
        adamw_kernel<bf16><<<1, 32, 0, st>>>((float*)p32 + done, tail16, (float*)m + done, (float*)v + done, (const bf16*)g + done,
                                             n - done, lr, beta1, beta2, eps, wd, bc1, bc2, (const float*)gscale, (const int*)skip);
    }
    return CHECK_LAUNCH();
  }
  int blocks = grid_for(n, 256);
  if (g_is_fp32)
    adamw_kernel<float><<<blocks, 256, 0, st>>>((float*)p32, (bf16*)p16, (float*)m, (float*)v, (const float*)g, n, lr,
                                                beta1, beta2, eps, wd, bc1, bc2, (const float*)gscale,
                                                (const int*)skip);
  else
    adamw_kernel<bf16><<<blocks, 256, 0, st>>>((float*)p32, (bf16*)p16, (float*)m, (float*)v, (const bf16*)g, n, lr,
                                               beta1, beta2, eps, wd, bc1, bc2, (const float*)gscale, (const int*)skip);
  return CHECK_LAUNCH();
}

int b200_muon_momentum(void* mom, const void* g, int g_is_fp32, void* out, void* sumsq, long n, float beta,
                       int nesterov, const void* gscale, float eps, cudaStream_t st) {
  if (n <= 0) return 0;
  cudaMemsetAsync(sumsq, 0, sizeof(float), st);
  if (n % 8 == 0 && aligned_to(mom, 16) && aligned_to(g, g_is_fp32 ? 16 : 8) && aligned_to(out, 16)) {
    // whole matrices: their element counts are multiples of 8 in every supported layout
    if (g_is_fp32)
      muon_momentum_vec_kernel<<<grid_for(n / 4, 256, 4), 256, 0, st>>>((float4*)mom, (const float4*)g, (bf16x4*)out, (float*)sumsq,
                                                                       n / 4, beta, nesterov, (const float*)gscale);
    else
      muon_momentum_vec_kernel<<<grid_for(n / 4, 256, 4), 256, 0, st>>>((float4*)mom, (const bf16x4*)g, (bf16x4*)out, (float*)sumsq,
                                                                       n / 4, beta, nesterov, (const float*)gscale);
    scale_by_norm_vec_kernel<<<grid_for(n / 8, 256, 4), 256, 0, st>>>((uint4*)out, (const float*)sumsq, n / 8, eps);
    return CHECK_LAUNCH();
  }
  int blocks = grid_for(n, 256, 4);
  if (g_is_fp32)
    muon_momentum_kernel<float><<<blocks, 256, 0, st>>>((float*)mom, (const float*)g, (bf16*)out, (float*)sumsq, n,
                                                        beta, nesterov, (const float*)gscale);
  else
    muon_momentum_kernel<bf16><<<blocks, 256, 0, st>>>((float*)mom, (const bf16*)g, (bf16*)out, (float*)sumsq, n, beta,
                                                       nesterov, (const float*)gscale);
  scale_by_norm_kernel<<<blocks, 256, 0, st>>>((bf16*)out, (const float*)sumsq, n, eps);
  return CHECK_LAUNCH();
}

int b200_muon_update(void* p32, void* p16, const void* o, long n, float lr, float wd, float scale, const void* skip,
                     cudaStream_t st) {
  if (n <= 0) return 0;
  if (n % 4 == 0 && aligned_to(p32, 16) && aligned_to(p16, 8) && aligned_to(o, 8)) {
    muon_update_vec_kernel<<<grid_for(n / 4, 256), 256, 0, st>>>((float4*)p32, (bf16x4*)p16, (const bf16x4*)o, n / 4, lr, wd, scale,
                                                                 (const int*)skip);
    return CHECK_LAUNCH();
  }
  muon_update_kernel<<<grid_for(n, 256), 256, 0, st>>>((float*)p32, (bf16*)p16, (const bf16*)o, n, lr, wd, scale,
                                                       (const int*)skip);
  return CHECK_LAUNCH();
}

int b200_ema(void* ema, const void* p, int p_is_fp32, long n, float decay, cudaStream_t st) {
  if (n <= 0) return 0;
  if (p_is_fp32) ema_kernel<float><<<grid_for(n, 256), 256, 0, st>>>((float*)ema, (const float*)p, n, decay);
  else ema_kernel<bf16><<<grid_for(n, 256), 256, 0, st>>>((float*)ema, (const bf16*)p, n, decay);
  return CHECK_LAUNCH();
}

// part: fp32 scratch of b200_num_partials() floats.  out[0] (+)= sum g^2.
int b200_sumsq(const void* g, int g_is_fp32, long n, void* part, void* out, int accumulate, cudaStream_t st) {
  int blocks = grid_for(n > 0 ? n : 1, 256, 2);
  if (g_is_fp32 && n >= 4 && aligned_to(g, 16)) {
    const long nv = n / 4;
    blocks = grid_for(nv, 256, 2);  // the partials scratch holds b200_num_partials() = 2 per SM
    sumsq_part_vec_kernel<<<blocks, 256, 0, st>>>((const float4*)g, (float*)part, nv, (const float*)g + nv * 4,
                                                  static_cast<int>(n - nv * 4));
    sumsq_finish_kernel<<<1, 256, 0, st>>>((const float*)part, (float*)out, blocks, accumulate);
    return CHECK_LAUNCH();
  }
  if (!g_is_fp32 && n >= 8 && aligned_to(g, 16)) {
    const long nv = n / 8;
    blocks = grid_for(nv, 256, 2);
    sumsq_part_bf16_kernel<<<blocks, 256, 0, st>>>((const uint4*)g, (float*)part, nv, (const bf16*)g + nv * 8, static_cast<int>(n - nv * 8));
    sumsq_finish_kernel<<<1, 256, 0, st>>>((const float*)part, (float*)out, blocks, accumulate);
    return CHECK_LAUNCH();
  }
  if (g_is_fp32) sumsq_part_kernel<float><<<blocks, 256, 0, st>>>((const float*)g, (float*)part, n);
  else sumsq_part_kernel<bf16><<<blocks, 256, 0, st>>>((const bf16*)g, (float*)part, n);
  sumsq_finish_kernel<<<1, 256, 0, st>>>((const float*)part, (float*)out, blocks, accumulate);
  return CHECK_LAUNCH();
}
int b200_clip_coef(const void* sumsq, void* norm_out, void* coef_out, void* skip_out, float max_norm,
                   const void* status, cudaStream_t st) {
  clip_coef_kernel<<<1, 1, 0, st>>>((const float*)sumsq, (float*)norm_out, (float*)coef_out, (int*)skip_out,
                                    max_norm, (const int*)status);
  return CHECK_LAUNCH();
}
int b200_scale(void* g, int g_is_fp32, long n, const void* coef, cudaStream_t st) {
  if (n <= 0) return 0;
  if (g_is_fp32) scale_kernel<float><<<grid_for(n, 256), 256, 0, st>>>((float*)g, n, (const float*)coef);
  else scale_kernel<bf16><<<grid_for(n, 256), 256, 0, st>>>((bf16*)g, n, (const float*)coef);
  return CHECK_LAUNCH();
}

// n_src / n_out: rows of the indexed tensor; an index beyond it raises kStatusBadIndex in *status and is skipped.
int b200_gather_rows(const void* src, const void* idx, void* out, long n_out, int H, long n_src, void* status,
                     cudaStream_t st) {
  if (n_out <= 0) return 0;
  if (H % 8) return -10;
  gather_rows_kernel<<<grid_for(n_out * (H / 8), 256), 256, 0, st>>>((const bf16*)src, (const int64_t*)idx, (bf16*)out,
                                                                     n_out, H, n_src, (int*)status);
  return CHECK_LAUNCH();
}
int b200_scatter_rows(const void* src, const void* idx, void* out, long n_src, int H, int add, long n_out, void* status,
                      cudaStream_t st) {
  if (n_src <= 0) return 0;
  if (H % 8) return -10;
  scatter_rows_kernel<<<grid_for(n_src * (H / 8), 256), 256, 0, st>>>((const bf16*)src, (const int64_t*)idx,
                                                                      (bf16*)out, n_src, H, add, n_out, (int*)status);
  return CHECK_LAUNCH();
}

int b200_ce_finalize(const void* stats, const void* logits, const void* labels, void* lse, void* loss, int rows,
                     int n_tiles, long ld, int V, int ignore_index, cudaStream_t st) {
  if (rows <= 0) return 0;
  ce_finalize_kernel<<<grid_for(static_cast<long>(rows) * 32, 256), 256, 0, st>>>(
      (const float2*)stats, (const bf16*)logits, (const int64_t*)labels, (float*)lse, (float*)loss, rows, n_tiles, ld,
      V, ignore_index);
  return CHECK_LAUNCH();
}
int b200_ce_dlogits(void* logits, const void* lse, const void* labels, const void* gscale, int rows, long ld, int V,
                    int ignore_index, cudaStream_t st) {
  if (rows <= 0) return 0;
  if (V % 8) return -10;
  int bx = (V / 8 + 255) / 256;
  if (bx > 16) bx = 16;
  int by = rows < 65535 ? rows : 65535;
  ce_dlogits_kernel<<<dim3(bx, by), 256, 0, st>>>((bf16*)logits, (const float*)lse, (const int64_t*)labels,
                                                  (const float*)gscale, rows, ld, V, ignore_index);
  return CHECK_LAUNCH();
}

}  // extern "C"

// ====================================================================================
// Allocation-free RMSNorm backward (see no_alloc.h for who needs it and for its limits).
// ====================================================================================
#include "no_alloc.h"

#include <mutex>

namespace b200 {

// Scratch for the per-CTA partial sums of dw.  File scope, device memory, part of the
// library image: no allocation at run time.  In host code this name is only a handle for
// cudaGetSymbolAddress, never a pointer a kernel could use.
static __device__ __align__(256) float g_noalloc_dw_part[B200_NOALLOC_MAX_PARTS * B200_NOALLOC_MAX_H];

constexpr int kNoAllocMaxDevices = 64;
static float* g_noalloc_ptr[kNoAllocMaxDevices] = {nullptr};
static std::mutex g_noalloc_mutex;

// Device address of the scratch array on the current device, resolved once per device.
static float* noalloc_scratch_for_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) return nullptr;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  if (g_noalloc_ptr[dev] == nullptr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_dw_part) != cudaSuccess || p == nullptr) return nullptr;
    g_noalloc_ptr[dev] = static_cast<float*>(p);
  }
  return g_noalloc_ptr[dev];
}

}  // namespace b200

extern "C" int b200_rmsnorm_bwd_noalloc(const void* dy, const void* x, const void* w, const void* rstd, void* dx,
                                        void* dw, int rows, int H, float w_offset, cudaStream_t st) {
  using namespace b200;
  if (rows <= 0) return 0;
  if (H % 8) return -10;
  if (H > B200_NOALLOC_MAX_H) return B200_NOALLOC_ERR_TOO_LARGE;
  float* part = noalloc_scratch_for_current_device();
  if (part == nullptr) return B200_NOALLOC_ERR_SETUP;
  int parts;
  if (H <= 512) {
    int blocks = num_sms() * 2 / 8;
    if (blocks < 1) blocks = 1;
    parts = blocks * 8;
    if (parts > B200_NOALLOC_MAX_PARTS) return B200_NOALLOC_ERR_TOO_LARGE;
    norm_bwd_warp_kernel<<<blocks, 256, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd,
                                                 (bf16*)dx, part, rows, H, w_offset);
  } else {
    parts = num_sms() * 2;
    if (parts > rows) parts = rows;
    if (parts > B200_NOALLOC_MAX_PARTS) parts = B200_NOALLOC_MAX_PARTS;
#define NOALLOC_BWD(T, V)                                                                                          \
  norm_bwd_kernel<T, V><<<parts, T, 0, st>>>((const bf16*)dy, (const bf16*)x, (const bf16*)w, (const float*)rstd, \
                                             nullptr, nullptr, (bf16*)dx, part, nullptr, rows, H, w_offset, 0)
    if (H <= 1024) NOALLOC_BWD(128, 1);
    else if (H <= 2048) NOALLOC_BWD(256, 1);
    else NOALLOC_BWD(256, 2);
#undef NOALLOC_BWD
  }
  if (cudaGetLastError() != cudaSuccess) return -4;
  // every partial row that is summed here was written by the launch above
  colsum(part, (float*)dw, parts, H, 0, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
