// Token-by-token generation: a few rows of activations against weights and cached keys / values that are read once.
//
// Every product here is bound by reading its weights, every attention by reading the cached rows, and a small model by
// the number of launches, so the path has five kernels per layer (seven above four rows, where the norms do not fit the
// products' prologue) and they
//   * start before the kernel in front of them has finished (programmatic dependent launch).  The products ask for their first
//     weights BEFORE they wait for it (weights never depend on it) and the attention for cached rows of earlier passes, so that
//     launch, ramp-up and DRAM latency of one kernel hide behind the tail of another; the row norm and the Gated-DeltaNet step
//     have nothing that they could load early and only launch early;
//   * read weights straight from global memory into mma.sync fragments (no shared-memory staging, see skinny_kernel);
//   * round to bf16 where the layer-by-layer path does (projection outputs, normalised rows, the residual stream) and evaluate
//     gates and decays as precisely as it does, so both paths compute the same numbers up to the order of fp32 sums.
//
//   skinny_kernel   y[M, N] = x[M, K] w[N, K]^T for M <= 64 rows, RMSNorm of x in its prologue (M <= 4), bias /
//                   residual add / SwiGLU in its epilogue, up to four weight matrices side by side along N
//   dec_attn_kernel per-head RMSNorm, rotary embedding, cache write and split-key attention of one new token per sequence
//   gdn_step_kernel one token of a Gated-DeltaNet layer: convolution tail, gates, state update, gated output norm
//   row_norm_kernel RMSNorm of M rows
//
// Reference counterpart: the same modules run one by one through transformers' generate
// (src/lmms_engine/models/aero_realtime/modeling_aero_realtime.py:700-1385 for the streaming loop).
// build: without --use_fast_math (gates and decays as the framework operations of the layer loop compute them; where the kernels of
// that path use the fast exponential and division, these are written out)
#include <atomic>

#include "common.cuh"

namespace b200 {

using bf16 = __nv_bfloat16;

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ uint4 ldg_stream(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ uint4 zero4() { return make_uint4(0u, 0u, 0u, 0u); }
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }
__device__ __forceinline__ float round_bf16(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
}
template <int kWarps>
__device__ __forceinline__ float cta_sum(float v, float* red) {
  v = warp_sum(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  const float t = warp_sum(lane < kWarps ? red[lane] : 0.f);
  __syncthreads();
  return t;
}

// ------------------------------------------------------------------------------------------------ skinny product
enum SkinnyMode : int { SK_PLAIN = 0, SK_RESID = 1, SK_SWIGLU = 2 };
constexpr int kSkSegs = 4;
constexpr int kSkNormRows = 4;   // rows that the fused norm prologue takes at most
constexpr int kSkWarps = 8;

struct SkinnyParams {
  const bf16* w[kSkSegs];        // weight matrices [rows, K], row stride ldw
  const bf16* bias[kSkSegs];     // or null
  int seg_end[kSkSegs];          // cumulative rows (SWIGLU: both matrices have N rows)
  int M, N, K;
  long ldw;
  const bf16* x;                 // [M, K], row stride ldx
  long ldx;
  const bf16* norm_w;            // fused norm: RMSNorm weight, or null
  float eps, norm_off;
  bf16* y;                       // PLAIN / SWIGLU output
  long ldy;
  bf16* res;                     // RESID: res = bf16(bf16(acc + bias) + res)
  long ldres;
};

// A CTA owns RT tiles of eight weight rows; its eight warps split K in 64-element steps (warp w takes steps w, w + 8, ...)
// and add up through shared memory.  The weights are the B operand of m16n8k16 (eight rows = n), the activations the A
// operand (MT tiles of sixteen rows).  Which k of the mma a loaded element stands for is free as long as A and B agree,
// so lane (g = lane / 4, t = lane % 4) loads 16 contiguous bytes of row g at k0 + 8 t and k0 + 32 + 8 t: full 128-byte
// lines of eight rows per warp and step, straight into fragments.
// RT = 1 below 17 rows: N / 8 CTAs are enough to fill the chip from N = 1024 on, and a row's slice of K per warp is short.
// From 17 rows on the activations (M x K) that every CTA reads from L2 outweigh eight weight rows, so RT grows to 2 (17 to 32
// rows) and 4 (33 rows and more), each as long as the grid still has a CTA for every SM (RT = 4 left 32 CTAs for the 1024
// output rows of a narrow model).
template <int RT, int MT, int MODE, bool NORM>
__global__ void __launch_bounds__(kSkWarps * 32) skinny_kernel(const __grid_constant__ SkinnyParams p) {
  extern __shared__ __align__(16) uint8_t dyn[];
  constexpr int U = RT == 1 ? 4 : 2;  // 64-element steps loaded at once per warp
  constexpr int kCols = RT * 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const int n_step = (p.K + 63) / 64;

  // weight row of every tile (null: past the end)
  const bf16* wrow[RT];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt) {
    if (MODE == SK_SWIGLU) {
      const int r = blockIdx.x * (4 * RT) + (rt % (RT / 2 > 0 ? RT / 2 : 1)) * 8;
      wrow[rt] = r < p.N ? p.w[rt < RT / 2 ? 0 : 1] + static_cast<size_t>(r + g) * p.ldw : nullptr;
    } else {
      const int r = blockIdx.x * kCols + rt * 8;
      wrow[rt] = nullptr;
      int lo = 0;
#pragma unroll
      for (int s = 0; s < kSkSegs; ++s) {
        if (r >= lo && r < p.seg_end[s]) wrow[rt] = p.w[s] + static_cast<size_t>(r - lo + g) * p.ldw;
        lo = p.seg_end[s];
      }
    }
  }

  uint4 wv[U][RT][2];
  auto load_w = [&](int step0) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (step0 + u * kSkWarps) * 64 + t * 8;
#pragma unroll
      for (int rt = 0; rt < RT; ++rt) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
          wv[u][rt][h] = (wrow[rt] != nullptr && k + h * 32 < p.K) ? ldg_stream(wrow[rt] + k + h * 32) : zero4();
      }
    }
  };
  load_w(warp);  // weights do not depend on the kernel in front
  pdl_go();
  pdl_wait();

  bf16* xs = reinterpret_cast<bf16*>(dyn);
  const long lds = p.K + 8;
  if (NORM) {
    __shared__ float red[kSkWarps];
    for (int m = 0; m < p.M; ++m) {
      float s2 = 0.f;
      for (int k = threadIdx.x * 8; k < p.K; k += kSkWarps * 256) {
        float v[8];
        unpack8(*reinterpret_cast<const uint4*>(p.x + m * p.ldx + k), v);
#pragma unroll
        for (int j = 0; j < 8; ++j) s2 += v[j] * v[j];
      }
      const float rstd = rsqrtf(cta_sum<kSkWarps>(s2, red) / p.K + p.eps);
      for (int k = threadIdx.x * 8; k < p.K; k += kSkWarps * 256) {
        float v[8], w8[8];
        unpack8(*reinterpret_cast<const uint4*>(p.x + m * p.ldx + k), v);
        unpack8(*reinterpret_cast<const uint4*>(p.norm_w + k), w8);
        uint4 o;
        uint32_t* ow = &o.x;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          ow[j] = pack_bf16x2(v[2 * j] * rstd * (w8[2 * j] + p.norm_off), v[2 * j + 1] * rstd * (w8[2 * j + 1] + p.norm_off));
        *reinterpret_cast<uint4*>(xs + m * lds + k) = o;
      }
    }
    __syncthreads();
  }

  float acc[RT][MT][4];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[rt][mt][j] = 0.f;

  for (int step0 = warp; step0 < n_step; step0 += U * kSkWarps) {
    if (step0 != warp) load_w(step0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (step0 + u * kSkWarps) * 64 + t * 8;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        uint4 xa[2], xb[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m0 = mt * 16 + g, m1 = m0 + 8, kk = k + h * 32;
          if (NORM) {
            xa[h] = (m0 < p.M && kk < p.K) ? *reinterpret_cast<const uint4*>(xs + m0 * lds + kk) : zero4();
            xb[h] = zero4();  // NORM takes at most kSkNormRows rows
          } else {
            xa[h] = (m0 < p.M && kk < p.K) ? *reinterpret_cast<const uint4*>(p.x + m0 * p.ldx + kk) : zero4();
            xb[h] = (m1 < p.M && kk < p.K) ? *reinterpret_cast<const uint4*>(p.x + m1 * p.ldx + kk) : zero4();
          }
        }
#pragma unroll
        for (int rt = 0; rt < RT; ++rt) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            mma_bf16(acc[rt][mt], xa[h].x, xb[h].x, xa[h].y, xb[h].y, wv[u][rt][h].x, wv[u][rt][h].y);
            mma_bf16(acc[rt][mt], xa[h].z, xb[h].z, xa[h].w, xb[h].w, wv[u][rt][h].z, wv[u][rt][h].w);
          }
        }
      }
    }
  }

  // add up the warps' slices of K: red[warp][row][col]
  if (NORM) __syncthreads();  // xs is overwritten
  float* red = reinterpret_cast<float*>(dyn);
  constexpr int kRows = MT * 16;
#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float* b = red + (static_cast<size_t>(warp) * kRows + mt * 16 + g) * kCols + rt * 8 + 2 * t;
      *reinterpret_cast<float2*>(b) = make_float2(acc[rt][mt][0], acc[rt][mt][1]);
      *reinterpret_cast<float2*>(b + 8 * kCols) = make_float2(acc[rt][mt][2], acc[rt][mt][3]);
    }
  __syncthreads();
  auto total = [&](int m, int c) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < kSkWarps; ++w) s += red[(w * kRows + m) * kCols + c];
    return s;
  };
  if (MODE == SK_SWIGLU) {
    constexpr int kOut = RT * 4;
    for (int i = threadIdx.x; i < p.M * kOut; i += kSkWarps * 32) {
      const int m = i / kOut, c = i % kOut;
      const int n = blockIdx.x * kOut + c;
      if (n >= p.N) continue;
      float gv = total(m, c), uv = total(m, c + kOut);
      if (p.bias[0] != nullptr) gv += __bfloat162float(p.bias[0][n]);
      if (p.bias[1] != nullptr) uv += __bfloat162float(p.bias[1][n]);
      gv = round_bf16(gv);
      uv = round_bf16(uv);
      p.y[m * p.ldy + n] = __float2bfloat16(__fdividef(gv, 1.0f + __expf(-gv)) * uv);
    }
  } else {
    for (int i = threadIdx.x; i < p.M * kCols; i += kSkWarps * 32) {
      const int m = i / kCols, c = i % kCols;
      const int n = blockIdx.x * kCols + c;
      if (n >= p.N) continue;
      float v = total(m, c);
      int lo = 0;
#pragma unroll
      for (int s = 0; s < kSkSegs; ++s) {
        if (n >= lo && n < p.seg_end[s] && p.bias[s] != nullptr) v += __bfloat162float(p.bias[s][n - lo]);
        lo = p.seg_end[s];
      }
      if (MODE == SK_RESID) {
        bf16* r = p.res + m * p.ldres + n;
        *r = __float2bfloat16(round_bf16(v) + __bfloat162float(*r));
      } else {
        p.y[m * p.ldy + n] = __float2bfloat16(v);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------------ row norm
// The kernel in front may still write `x` when this one starts, so `x` is not declared __restrict__: the compiler could then
// read it through the non-coherent path or above the wait.  Only the weight is unchanged for the whole launch.
__global__ void __launch_bounds__(256) row_norm_kernel(const bf16* x, const bf16* __restrict__ w, bf16* y, int K, long ldx,
                                                       long ldy, float eps, float off) {
  __shared__ float red[8];
  pdl_go();
  pdl_wait();
  const bf16* xr = x + blockIdx.x * ldx;
  float s2 = 0.f;
  for (int k = threadIdx.x * 8; k < K; k += 2048) {
    float v[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + k), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) s2 += v[j] * v[j];
  }
  const float rstd = rsqrtf(cta_sum<8>(s2, red) / K + eps);
  for (int k = threadIdx.x * 8; k < K; k += 2048) {
    float v[8], w8[8];
    unpack8(*reinterpret_cast<const uint4*>(xr + k), v);
    unpack8(*reinterpret_cast<const uint4*>(w + k), w8);
    uint4 o;
    uint32_t* ow = &o.x;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      ow[j] = pack_bf16x2(v[2 * j] * rstd * (w8[2 * j] + off), v[2 * j + 1] * rstd * (w8[2 * j + 1] + off));
    *reinterpret_cast<uint4*>(y + blockIdx.x * ldy + k) = o;
  }
}

// ------------------------------------------------------------------------------------------------ attention of one new token
constexpr int kDecSeqs = 64;

struct DecAttnParams {
  const bf16* proj;              // [n_seq, ld]: query / gate / key / value projections of the new tokens
  long ld;
  int q_off, q_hs, gate_off;     // query head h at q_off + h * q_hs; its gate at gate_off + h * q_hs (gate_off < 0: none)
  int k_off, v_off;
  const bf16* qn;                // per-head RMSNorm weights, or null
  const bf16* kn;
  float norm_off, eps;
  const float* cos;              // [n_seq, rot] fp32
  const float* sin;
  int rot;
  bf16* kc;                      // cache slabs [rows, n_kv, D]
  bf16* vc;
  int n_kv, group;
  float scale_log2;
  int window;                    // keys further back than this are not seen (< 0: all)
  int splits;
  float* ws;                     // partial results [n_seq, n_kv, splits, group, D], then their (max, sum) [..., 2]
  int* count;                    // [n_seq, n_kv] arrivals; returned to zero
  bf16* out;                     // [n_seq, n_kv * group * D]
  long ldo;
  int base[kDecSeqs], have[kDecSeqs];  // first cache row and cached rows of every sequence before this token
};

// One warp normalises and rotates one head (D elements, element lane + 32 i in register i); `s` holds the head as bf16.
template <int D>
__device__ __forceinline__ void head_norm_rope(const bf16* src, const bf16* w, float off, float eps, const float* c,
                                               const float* s, int rot, bf16* dst, int lane) {
  float v[D / 32];
  float s2 = 0.f;
#pragma unroll
  for (int i = 0; i < D / 32; ++i) {
    v[i] = __bfloat162float(src[lane + 32 * i]);
    s2 += v[i] * v[i];
  }
  if (w != nullptr) {
    const float rstd = rsqrtf(warp_sum(s2) / D + eps);
#pragma unroll
    for (int i = 0; i < D / 32; ++i) v[i] = v[i] * rstd * (__bfloat162float(w[lane + 32 * i]) + off);
  }
#pragma unroll
  for (int i = 0; i < D / 32; ++i) dst[lane + 32 * i] = __float2bfloat16(v[i]);
  __syncwarp();
  const int half = rot / 2;
#pragma unroll
  for (int i = 0; i < D / 32; ++i) {
    const int d = lane + 32 * i;
    if (d < half) v[i] = __bfloat162float(dst[d]) * c[d] - __bfloat162float(dst[d + half]) * s[d];
    else if (d < rot) v[i] = __bfloat162float(dst[d]) * c[d] + __bfloat162float(dst[d - half]) * s[d];
    else v[i] = __bfloat162float(dst[d]);
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < D / 32; ++i) dst[lane + 32 * i] = __float2bfloat16(v[i]);
}

// Grid (splits, n_kv, n_seq), four warps.  The query heads that share a key head are the rows of one m16n8k16 tile
// (QROWS = 8: rows 8..15 stay zero).  A warp walks every fourth block of sixteen keys of its CTA's share with its own
// running maximum; keys go from global memory straight into fragments (the same free choice of k as in skinny_kernel),
// values through two warp-private shared-memory tiles that ldmatrix reads transposed.  The shares of a key head are
// combined by the CTA that finishes last.  Bound by reading the cached rows: a share is at least 64 keys, and there are
// as many shares as fill the chip about twice.
template <int D, int QROWS>
__global__ void __launch_bounds__(128) dec_attn_kernel(const __grid_constant__ DecAttnParams p) {
  constexpr int NC = D / 32;                 // 32-element chunks of a head
  constexpr int NT = D / 8;                  // eight-wide output tiles
  constexpr int RH = QROWS / 8;
  extern __shared__ __align__(16) uint8_t dyn[];
  bf16* sQ = reinterpret_cast<bf16*>(dyn);                          // [16][D]
  bf16* sK = sQ + 16 * D;                                           // [D] the new key
  bf16* sV = sK + D;                                                // [4 warps][2][16][D]
  float* sO = reinterpret_cast<float*>(sV);                         // [4][QROWS][D] after the loop
  float* sML = reinterpret_cast<float*>(sV + 4 * 2 * 16 * D);       // [4][QROWS][2]
  int* sLast = reinterpret_cast<int*>(sML + 4 * QROWS * 2);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int split = blockIdx.x, kvh = blockIdx.y, seq = blockIdx.z;
  const int total = p.have[seq] + 1;
  const int k_min = p.window >= 0 ? max(0, total - 1 - p.window) : 0;
  int share = (total - k_min + p.splits - 1) / p.splits;
  share = (share + 63) / 64 * 64;
  const int lo = min(total, k_min + split * share), hi = min(total, lo + share);
  const bool last_share = lo < hi && hi == total;
  const long row_ld = static_cast<long>(p.n_kv) * D;
  const size_t head_off = static_cast<size_t>(p.base[seq]) * row_ld + static_cast<size_t>(kvh) * D;
  bf16* kc = p.kc + head_off;
  bf16* vc = p.vc + head_off;

  // The cached rows do not depend on the kernel in front of this one: a warp whose first block holds older keys only loads
  // it before the wait.
  bf16* vt = sV + warp * 2 * 16 * D;
  const int n_blk = (hi - lo + 15) / 16;
  uint4 kf[2][NC];
  auto load_k = [&](int b) {
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int key = min(lo + b * 16 + n * 8 + g, hi - 1);
#pragma unroll
      for (int c = 0; c < NC; ++c) kf[n][c] = *reinterpret_cast<const uint4*>(kc + key * row_ld + c * 32 + t * 8);
    }
  };
  auto load_v = [&](int b, int buf) {  // 16-byte pieces, piece index xor key so that ldmatrix rows fall on distinct banks
    constexpr int kPieces = D / 8;
#pragma unroll
    for (int i = 0; i < 16 * kPieces / 32; ++i) {
      const int idx = i * 32 + lane, r = idx / kPieces, c = idx % kPieces;
      const int key = min(lo + b * 16 + r, hi - 1);
      const uint32_t dst = smem_u32(vt + buf * 16 * D + r * D + ((c ^ (r & 7)) * 8));
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(vc + key * row_ld + c * 8) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const bool early = warp < n_blk && lo + (warp + 1) * 16 <= total - 1;
  if (early) {
    load_v(warp, 0);
    load_k(warp);
  }

  pdl_go();
  pdl_wait();
  const bf16* pr = p.proj + seq * p.ld;
  const float* cs = p.cos + static_cast<size_t>(seq) * p.rot;
  const float* sn = p.sin + static_cast<size_t>(seq) * p.rot;
  for (int i = threadIdx.x; i < 16 * D / 8; i += 128) reinterpret_cast<uint4*>(sQ)[i] = zero4();
  __syncthreads();
  for (int h = warp; h < p.group + 1; h += 4) {
    if (h < p.group)
      head_norm_rope<D>(pr + p.q_off + static_cast<long>(kvh * p.group + h) * p.q_hs, p.qn, p.norm_off, p.eps, cs, sn, p.rot, sQ + h * D, lane);
    else if (last_share)
      head_norm_rope<D>(pr + p.k_off + kvh * D, p.kn, p.norm_off, p.eps, cs, sn, p.rot, sK, lane);
  }
  __syncthreads();
  if (last_share && threadIdx.x < D / 8) {
    const long at = static_cast<long>(total - 1) * row_ld + threadIdx.x * 8;
    *reinterpret_cast<uint4*>(kc + at) = reinterpret_cast<const uint4*>(sK)[threadIdx.x];
    *reinterpret_cast<uint4*>(vc + at) = *reinterpret_cast<const uint4*>(pr + p.v_off + kvh * D + threadIdx.x * 8);
  }
  __syncthreads();

  uint4 qf[NC][RH];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int r = 0; r < RH; ++r) qf[c][r] = *reinterpret_cast<const uint4*>(sQ + (g + 8 * r) * D + c * 32 + t * 8);

  float o[NT][4];
#pragma unroll
  for (int j = 0; j < NT; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
  if (warp < n_blk && !early) {
    load_v(warp, 0);
    load_k(warp);
  }
  int buf = 0;
  for (int b = warp; b < n_blk; b += 4, buf ^= 1) {
    float s[2][4];
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const uint4 qa = qf[c][0], qb = RH == 2 ? qf[c][RH - 1] : zero4();
        mma_bf16(s[n], qa.x, qb.x, qa.y, qb.y, kf[n][c].x, kf[n][c].y);
        mma_bf16(s[n], qa.z, qb.z, qa.w, qb.w, kf[n][c].z, kf[n][c].w);
      }
    }
    const bool more = b + 4 < n_blk;
    if (more) {
      load_k(b + 4);
      load_v(b + 4, buf ^ 1);
    }
    uint32_t pk[2][2];
#pragma unroll
    for (int r = 0; r < RH; ++r) {
      float m = mx[r];
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          float& v = s[n][2 * r + e];
          v = lo + b * 16 + n * 8 + 2 * t + e < hi ? v * p.scale_log2 : -INFINITY;
          m = fmaxf(m, v);
        }
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
      const float alpha = fast_exp2(mx[r] - m);  // the block holds at least one visible key, so m is finite
      mx[r] = m;
      float add = 0.f;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        const float e0 = fast_exp2(s[n][2 * r] - m), e1 = fast_exp2(s[n][2 * r + 1] - m);
        add += e0 + e1;
        pk[n][r] = pack_bf16x2(e0, e1);
      }
      sum[r] = sum[r] * alpha + add;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        o[j][2 * r] *= alpha;
        o[j][2 * r + 1] *= alpha;
      }
    }
    if (RH == 1) pk[0][1] = pk[1][1] = 0u;
    if (more) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int j = 0; j < NT; j += 2) {
      // four 8 x 8 tiles: keys 0-7 / 8-15 of output tile j, then of j + 1
      const int r = lane & 15, c = j + (lane >> 4);
      const uint32_t src = smem_u32(vt + buf * 16 * D + r * D + ((c ^ (r & 7)) * 8));
      uint32_t b0, b1, b2, b3;
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                   : "=r"(b0), "=r"(b1), "=r"(b2), "=r"(b3)
                   : "r"(src)
                   : "memory");
      mma_bf16(o[j], pk[0][0], pk[0][1], pk[1][0], pk[1][1], b0, b1);
      mma_bf16(o[j + 1], pk[0][0], pk[0][1], pk[1][0], pk[1][1], b2, b3);
    }
    __syncwarp();  // the tile is refilled by the next iteration's prefetch
  }

  // the four warps, then the shares
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RH; ++r) {
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    const int row = g + 8 * r;
    if (t == 0) {
      sML[(warp * QROWS + row) * 2] = mx[r];
      sML[(warp * QROWS + row) * 2 + 1] = sum[r];
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
      *reinterpret_cast<float2*>(sO + (warp * QROWS + row) * D + j * 8 + 2 * t) = make_float2(o[j][2 * r], o[j][2 * r + 1]);
  }
  __syncthreads();
  auto store = [&](int h, int d, float v) {
    float r = round_bf16(v);
    if (p.gate_off >= 0)
      r = r * sigmoid_f(__bfloat162float(pr[p.gate_off + static_cast<long>(kvh * p.group + h) * p.q_hs + d]));
    p.out[seq * p.ldo + static_cast<long>(kvh * p.group + h) * D + d] = __float2bfloat16(r);
  };
  const size_t share0 = static_cast<size_t>(seq * p.n_kv + kvh) * p.splits * p.group;   // (share, head) pairs in front
  float* wo = p.ws + share0 * D;
  float2* wml = reinterpret_cast<float2*>(p.ws + static_cast<size_t>(gridDim.z) * p.n_kv * p.splits * p.group * D) + share0;
  for (int i = threadIdx.x; i < p.group * D; i += 128) {
    const int h = i / D, d = i % D;
    float m = -INFINITY;
#pragma unroll
    for (int w = 0; w < 4; ++w) m = fmaxf(m, sML[(w * QROWS + h) * 2]);
    float l = 0.f, v = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const float mw = sML[(w * QROWS + h) * 2];
      if (mw > -INFINITY) {
        const float f = fast_exp2(mw - m);
        l += f * sML[(w * QROWS + h) * 2 + 1];
        v += f * sO[(w * QROWS + h) * D + d];
      }
    }
    if (p.splits == 1) {
      store(h, d, __fdividef(v, l));
    } else {
      wo[(split * p.group + h) * D + d] = v;
      if (d == 0) wml[split * p.group + h] = make_float2(m, l);
    }
  }
  if (p.splits == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    int* c = p.count + seq * p.n_kv + kvh;
    const int prev = atomicAdd(c, 1);
    *sLast = prev == p.splits - 1;
    if (*sLast) *c = 0;  // nobody else touches it before the next launch
  }
  __syncthreads();
  if (!*sLast) return;
  __threadfence();
  // A warp per head, four columns per lane (two shares side by side for D = 64): the loads of a share depend on nothing, so
  // eight of them are in flight.  One thread per element instead walked all shares once for the maximum and once for the sum:
  // 64 shares x 7 heads took longer than the attention itself.
  constexpr int LR = D / 4, SG = 32 / LR;
  const int sg = lane / LR, d0 = (lane % LR) * 4;
  for (int h = warp; h < p.group; h += 4) {
    float2 ml[2] = {make_float2(-INFINITY, 0.f), make_float2(-INFINITY, 0.f)};   // shares lane and lane + 32 (at most 64)
#pragma unroll
    for (int i = 0; i < 2; ++i)
      if (lane + 32 * i < p.splits) ml[i] = __ldcg(wml + (lane + 32 * i) * p.group + h);
    const float m = warp_max(fmaxf(ml[0].x, ml[1].x));
    const float f0 = fast_exp2(ml[0].x - m), f1 = fast_exp2(ml[1].x - m);  // an empty share has m = -inf: weight 0
    const float l = warp_sum(f0 * ml[0].y + f1 * ml[1].y);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int s0 = 0; s0 < p.splits; s0 += SG) {
      const int s = s0 + sg;
      const float g0 = __shfl_sync(0xffffffffu, f0, s & 31), g1 = __shfl_sync(0xffffffffu, f1, s & 31);
      const float w = s < 32 ? g0 : g1;
      if (s < p.splits) {
        const float4 o4 = __ldcg(reinterpret_cast<const float4*>(wo + (s * p.group + h) * D + d0));
        v.x += w * o4.x; v.y += w * o4.y; v.z += w * o4.z; v.w += w * o4.w;
      }
    }
    if (SG == 2) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, 16); v.y += __shfl_xor_sync(0xffffffffu, v.y, 16);
      v.z += __shfl_xor_sync(0xffffffffu, v.z, 16); v.w += __shfl_xor_sync(0xffffffffu, v.w, 16);
    }
    if (sg == 0) {
      const float inv = __fdividef(1.f, l);
      store(h, d0, v.x * inv); store(h, d0 + 1, v.y * inv); store(h, d0 + 2, v.z * inv); store(h, d0 + 3, v.w * inv);
    }
  }
}

// ------------------------------------------------------------------------------------------------ Gated-DeltaNet, one token
constexpr int kGdnD = 128;  // key and value head dim

struct GdnStepParams {
  const bf16* proj;              // [n_seq, ld]: convolution input (q | k | v), z, b, a
  long ld;
  int key_dim, z_off, b_off, a_off;
  int hk, hv, conv_dim, taps;
  const bf16* conv_w;            // [conv_dim, taps]
  const bf16* A_log;             // [hv]
  const bf16* dt_bias;           // [hv]
  const bf16* norm_w;            // [128]
  float eps;
  bf16* out;                     // [n_seq, hv * 128]
  long ldo;
  const bf16* tail_in[kDecSeqs];   // [taps - 1, conv_dim] rows that went into the convolution before this token
  bf16* tail_out[kDecSeqs];        // another buffer: heads that share key channels read the old rows
  const float* state_in[kDecSeqs]; // [hv, 128, 128]
  float* state_out[kDecSeqs];      // another buffer: whoever holds the state before this token keeps it
};

// One CTA per (value head, sequence); thread (half, v) keeps 64 rows of column v of the state in registers, so the state
// is read and written once, coalesced along v.  Bound by the latency of that chain, not by its 64 KB.
__global__ void __launch_bounds__(256) gdn_step_kernel(const __grid_constant__ GdnStepParams p) {
  __shared__ float sq[kGdnD], sk[kGdnD], sv[kGdnD], part[2][kGdnD], part2[2][kGdnD], red[8];
  const int vh = blockIdx.x, seq = blockIdx.y, tid = threadIdx.x;
  const int col = tid & (kGdnD - 1), half = tid >> 7;
  const size_t at = (static_cast<size_t>(vh) * kGdnD + half * 64) * kGdnD + col;
  const float* S = p.state_in[seq] + at;
  float* So = p.state_out[seq] + at;
  pdl_go();
  pdl_wait();
  float st[64];
#pragma unroll
  for (int i = 0; i < 64; ++i) st[i] = S[i * kGdnD];
  const bf16* pr = p.proj + seq * p.ld;
  const int rep = p.hv / p.hk, qh = vh / rep;
  for (int i = tid; i < 3 * kGdnD; i += 256) {
    const int which = i / kGdnD, d = i % kGdnD;
    const int ch = which == 0 ? qh * kGdnD + d : (which == 1 ? p.key_dim + qh * kGdnD + d : 2 * p.key_dim + vh * kGdnD + d);
    const float cur = __bfloat162float(pr[ch]);
    const bf16* w = p.conv_w + static_cast<size_t>(ch) * p.taps;
    const bf16* ti = p.tail_in[seq];
    bf16* to = p.tail_out[seq];
    const bool keeper = which == 2 || vh % rep == 0;
    float acc = cur * __bfloat162float(w[p.taps - 1]);
    for (int j = 1; j < p.taps; ++j) {
      const bf16 old = ti[static_cast<size_t>(p.taps - 1 - j) * p.conv_dim + ch];
      acc += __bfloat162float(old) * __bfloat162float(w[p.taps - 1 - j]);
      if (keeper && p.taps - 2 - j >= 0) to[static_cast<size_t>(p.taps - 2 - j) * p.conv_dim + ch] = old;
    }
    if (keeper) to[static_cast<size_t>(p.taps - 2) * p.conv_dim + ch] = pr[ch];
    const float y = round_bf16(__fdividef(acc, 1.0f + __expf(-acc)));
    (which == 0 ? sq : (which == 1 ? sk : sv))[d] = y;
  }
  __syncthreads();
  const float kq = half == 0 ? sq[col] : sk[col];
  // sums of squares of q (first half of the threads) and k (second half)
  const float ss = warp_sum(kq * kq);
  if ((tid & 31) == 0) red[tid >> 5] = ss;
  __syncthreads();
  const float qn = rsqrtf(red[0] + red[1] + red[2] + red[3] + 1e-6f) * rsqrtf(static_cast<float>(kGdnD));
  const float kn = rsqrtf(red[4] + red[5] + red[6] + red[7] + 1e-6f);
  const float beta = round_bf16(sigmoid_f(__bfloat162float(pr[p.b_off + vh])));
  const float a = __bfloat162float(pr[p.a_off + vh]) + __bfloat162float(p.dt_bias[vh]);
  const float sp = a > 20.f ? a : log1pf(expf(a));
  const float decay = expf(-expf(__bfloat162float(p.A_log[vh])) * sp);
  float ks = 0.f;
#pragma unroll
  for (int i = 0; i < 64; ++i) {
    st[i] *= decay;
    ks += sk[half * 64 + i] * st[i];
  }
  part[half][col] = ks * kn;
  __syncthreads();
  const float delta = (sv[col] - part[0][col] - part[1][col]) * beta;
  float oo = 0.f;
#pragma unroll
  for (int i = 0; i < 64; ++i) {
    st[i] += sk[half * 64 + i] * kn * delta;
    oo += sq[half * 64 + i] * st[i];
    So[i * kGdnD] = st[i];
  }
  part2[half][col] = oo * qn;
  __syncthreads();
  const float o = round_bf16(part2[0][col] + part2[1][col]);
  const float s2 = warp_sum(o * o);
  if ((tid & 31) == 0) red[tid >> 5] = s2;
  __syncthreads();
  if (half == 0) {
    const float rstd = rsqrtf((red[0] + red[1] + red[2] + red[3]) / kGdnD + p.eps);
    const float n = round_bf16(o * rstd * __bfloat162float(p.norm_w[col]));
    const float z = __bfloat162float(pr[p.z_off + vh * kGdnD + col]);
    p.out[seq * p.ldo + static_cast<long>(vh) * kGdnD + col] = __float2bfloat16(n * (z / (1.0f + expf(-z))));
  }
}

// ------------------------------------------------------------------------------------------------ host side
// `early`: this kernel may start while the one in front of it in the stream still runs.  Only inside the chain of
// b200_decode_layers, where that kernel never writes weights; a caller's weight may come straight from another kernel.
template <typename P>
static int launch_k(void (*k)(const P), dim3 grid, int threads, size_t smem, cudaStream_t st, const P& p, bool early) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, p) == cudaSuccess ? 0 : -4;
}

// Dynamic shared memory beyond the default limit has to be asked for once per kernel and device.  The amount is always the
// kernel's largest, so that threads with different sizes do not lower it for one another; two that come first at the same time
// ask for the same.
struct SmemOptIn {
  std::atomic<unsigned long long> done{0};   // a bit per device
  template <typename K>
  int ask(K kernel, size_t bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -3;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess) return -3;
    done.fetch_or(bit, std::memory_order_release);
    return 0;
  }
};

constexpr size_t kNormRowsBytes = 96 * 1024;   // most that the rows of the fused norm may take
static bool norm_fits(int M, int K) { return M <= kSkNormRows && static_cast<size_t>(M) * (K + 8) * 2 <= kNormRowsBytes; }

template <int RT, int MT, int MODE, bool NORM>
static int launch_skinny(const SkinnyParams& p, cudaStream_t st, bool early) {
  constexpr size_t kParts = static_cast<size_t>(kSkWarps) * MT * 16 * RT * 8 * 4;
  size_t smem = kParts;
  if (NORM) {
    const size_t xs = static_cast<size_t>(p.M) * (p.K + 8) * 2;
    if (xs > smem) smem = xs;
  }
  static SmemOptIn opt;
  if (opt.ask(skinny_kernel<RT, MT, MODE, NORM>, NORM && kNormRowsBytes > kParts ? kNormRowsBytes : kParts) != 0) return -3;
  const int per = MODE == SK_SWIGLU ? RT * 4 : RT * 8;
  return launch_k(skinny_kernel<RT, MT, MODE, NORM>, dim3((p.N + per - 1) / per), kSkWarps * 32, smem, st, p, early);
}

static int num_sms() {
  static std::atomic<int> sms{0};
  int n = sms.load(std::memory_order_relaxed);
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    sms.store(n, std::memory_order_relaxed);
  }
  return n;
}

template <int MT, int MODE>
static int wide(const SkinnyParams& p, cudaStream_t st, bool early) {
  constexpr int per = MODE == SK_SWIGLU ? 4 : 8;   // output rows per weight tile
  const int sms = num_sms();
  if constexpr (MT > 2) {
    if (p.N >= sms * per * 4) return launch_skinny<4, MT, MODE, false>(p, st, early);
  }
  if (MODE == SK_SWIGLU || p.N >= sms * per * 2) return launch_skinny<2, MT, MODE, false>(p, st, early);
  return launch_skinny<MODE == SK_SWIGLU ? 2 : 1, MT, MODE, false>(p, st, early);
}

template <int MODE>
static int skinny(const SkinnyParams& p, cudaStream_t st, bool early = true) {
  constexpr int R1 = MODE == SK_SWIGLU ? 2 : 1;
  if (p.norm_w != nullptr) return launch_skinny<R1, 1, MODE, true>(p, st, early);
  if (p.M <= 16) return launch_skinny<R1, 1, MODE, false>(p, st, early);
  if (p.M <= 32) return wide<2, MODE>(p, st, early);
  if (p.M <= 48) return wide<3, MODE>(p, st, early);
  return wide<4, MODE>(p, st, early);
}

static int row_norm(const bf16* x, const bf16* w, bf16* y, int M, int K, float eps, float off, cudaStream_t st) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(M);
  cfg.blockDim = dim3(256);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, row_norm_kernel, x, w, y, K, static_cast<long>(K), static_cast<long>(K), eps, off) == cudaSuccess ? 0 : -4;
}

template <int D, int QROWS>
static int launch_dec_attn(const DecAttnParams& p, int n_seq, cudaStream_t st) {
  constexpr size_t smem = (16 * D + D + 4 * 2 * 16 * D) * 2 + 4 * QROWS * 2 * 4 + 16;
  static_assert(4 * QROWS * D * 4 <= 4 * 2 * 16 * D * 2, "outputs of the warps reuse the value tiles");
  static SmemOptIn opt;
  if (opt.ask(dec_attn_kernel<D, QROWS>, smem) != 0) return -3;
  return launch_k(dec_attn_kernel<D, QROWS>, dim3(p.splits, p.n_kv, n_seq), 128, smem, st, p, true);
}

}  // namespace b200

using namespace b200;

extern "C" {

// y[M, N] = x[M, K] w[N, K]^T (+ bias) for M <= 64; K and N multiples of 8, 16-byte aligned rows.
int b200_skinny_linear(const void* x, const void* w, const void* bias, void* y, int M, int N, int K, long ldx, long ldw,
                       long ldy, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (M > 64 || ((N | K) & 7) || ((ldx | ldw | ldy) & 7)) return -10;
  SkinnyParams p{};
  p.w[0] = static_cast<const bf16*>(w);
  p.bias[0] = static_cast<const bf16*>(bias);
  for (int s = 0; s < kSkSegs; ++s) p.seg_end[s] = N;
  p.M = M; p.N = N; p.K = K;
  p.ldw = ldw;
  p.x = static_cast<const bf16*>(x);
  p.ldx = ldx;
  p.y = static_cast<bf16*>(y);
  p.ldy = ldy;
  return skinny<SK_PLAIN>(p, st, false);
}

// Work buffer of b200_decode_layers in bytes (256-byte pieces): projections | mixer output | MLP hidden | normalised rows |
// attention shares.
static size_t up256(size_t n) { return (n + 255) & ~static_cast<size_t>(255); }

// All layers of a decoder for ONE new token per sequence; `res` [M, H] holds the embeddings and becomes the residual
// stream, `hidden` [M, H] receives the final norm.
//   lw     per layer 24 pointers:
//          0 input norm | 1..4 projection weights | 5..8 their biases | 9 q norm | 10 k norm | 11 output projection |
//          12 post norm | 13 gate | 14 up | 15 down | 16 key slab | 17 value slab |
//          19 output bias | (linear attention) 9 conv weight | 10 A_log | 16 dt_bias | 17 gated norm weight
//   lt     per layer: 0 attention, 1 attention with an output gate, 2 Gated-DeltaNet
//   gdn    per linear-attention layer and sequence: tail in, tail out, state in, state out
//   dims   0 M 1 H 2 heads 3 kv heads 4 head dim 5 rotary dim 6 intermediate 7 window 8 splits
//          9 key heads 10 value heads 11 taps (linear attention)
int b200_decode_layers(const unsigned long long* lw, const int* lt, int n_layers, const int* dims, const int* base,
                       const int* have, const unsigned long long* gdn, float eps, float norm_off, float scale,
                       const void* cosb, const void* sinb, void* res, void* hidden, const void* final_norm, void* work,
                       long work_bytes, void* shares, void* count, cudaStream_t st) {
  const int M = dims[0], H = dims[1], nq = dims[2], nkv = dims[3], D = dims[4], rot = dims[5], I = dims[6];
  const int hk = dims[9], hv = dims[10], taps = dims[11];
  if (M <= 0 || M > kDecSeqs) return -10;
  bool any_gdn = false, any_attn = false, any_gate = false;
  for (int l = 0; l < n_layers; ++l) {
    any_gdn |= lt[l] == 2;
    any_attn |= lt[l] != 2;
    any_gate |= lt[l] == 1;
  }
  if (any_attn && ((D != 64 && D != 128) || nq % nkv || nq / nkv > 16)) return -11;
  const int key_dim = hk * kGdnD, val_dim = hv * kGdnD;
  int np = 0, no = 0;
  if (any_attn) { np = nq * D * (any_gate ? 2 : 1) + 2 * nkv * D; no = nq * D; }
  if (any_gdn) {
    const int g = 2 * key_dim + 2 * val_dim + 2 * hv;
    if (g > np) np = g;
    if (val_dim > no) no = val_dim;
  }
  uint8_t* wp = static_cast<uint8_t*>(work);
  bf16* proj = reinterpret_cast<bf16*>(wp); wp += up256(static_cast<size_t>(M) * np * 2);
  bf16* mix = reinterpret_cast<bf16*>(wp); wp += up256(static_cast<size_t>(M) * no * 2);
  bf16* mlp = reinterpret_cast<bf16*>(wp); wp += up256(static_cast<size_t>(M) * I * 2);
  bf16* xn = reinterpret_cast<bf16*>(wp); wp += up256(static_cast<size_t>(M) * H * 2);
  if (wp - static_cast<uint8_t*>(work) > work_bytes) return -12;
  bf16* r = static_cast<bf16*>(res);
  const bool fuse = norm_fits(M, H);
  int gi = 0;

  auto ptr = [&](int l, int i) { return reinterpret_cast<const bf16*>(lw[static_cast<size_t>(l) * 24 + i]); };
  auto input = [&](SkinnyParams& p, const bf16* nw) -> int {  // the product reads the normalised residual stream
    p.M = M; p.K = H; p.ldw = H;
    if (fuse) {
      p.x = r; p.ldx = H;
      p.norm_w = nw; p.eps = eps; p.norm_off = norm_off;
      return 0;
    }
    p.x = xn; p.ldx = H;
    return row_norm(r, nw, xn, M, H, eps, norm_off, st);
  };
  for (int l = 0; l < n_layers; ++l) {
    int rc = 0;
    SkinnyParams p{};
    if ((rc = input(p, ptr(l, 0))) != 0) return rc;
    int rows[kSkSegs] = {0, 0, 0, 0};
    if (lt[l] == 2) { rows[0] = 2 * key_dim + val_dim; rows[1] = val_dim; rows[2] = hv; rows[3] = hv; }
    else { rows[0] = nq * D * (lt[l] == 1 ? 2 : 1); rows[1] = nkv * D; rows[2] = nkv * D; }
    int at = 0;
    for (int s = 0; s < kSkSegs; ++s) {
      p.w[s] = ptr(l, 1 + s);
      p.bias[s] = ptr(l, 5 + s);
      if (rows[s] & 7) return -13;  // a tile of eight weight rows belongs to one matrix
      at += rows[s];
      p.seg_end[s] = at;
    }
    p.N = at;
    p.y = proj; p.ldy = at;
    if ((rc = skinny<SK_PLAIN>(p, st)) != 0) return rc;
    int mix_n = nq * D;
    if (lt[l] == 2) {
      mix_n = val_dim;
      GdnStepParams q{};
      q.proj = proj; q.ld = at;
      q.key_dim = key_dim; q.z_off = 2 * key_dim + val_dim; q.b_off = q.z_off + val_dim; q.a_off = q.b_off + hv;
      q.hk = hk; q.hv = hv; q.conv_dim = 2 * key_dim + val_dim; q.taps = taps;
      q.conv_w = ptr(l, 9); q.A_log = ptr(l, 10); q.dt_bias = ptr(l, 16); q.norm_w = ptr(l, 17);
      q.eps = eps;
      q.out = mix; q.ldo = val_dim;
      for (int s = 0; s < M; ++s) {
        const unsigned long long* e = gdn + (static_cast<size_t>(gi) * M + s) * 4;
        q.tail_in[s] = reinterpret_cast<const bf16*>(e[0]);
        q.tail_out[s] = reinterpret_cast<bf16*>(e[1]);
        q.state_in[s] = reinterpret_cast<const float*>(e[2]);
        q.state_out[s] = reinterpret_cast<float*>(e[3]);
      }
      ++gi;
      if ((rc = launch_k(gdn_step_kernel, dim3(hv, M), 256, 0, st, q, true)) != 0) return rc;
    } else {
      DecAttnParams a{};
      a.proj = proj; a.ld = at;
      a.q_off = 0; a.q_hs = lt[l] == 1 ? 2 * D : D; a.gate_off = lt[l] == 1 ? D : -1;
      a.k_off = rows[0]; a.v_off = rows[0] + rows[1];
      a.qn = ptr(l, 9); a.kn = ptr(l, 10); a.norm_off = norm_off; a.eps = eps;
      a.cos = static_cast<const float*>(cosb); a.sin = static_cast<const float*>(sinb); a.rot = rot;
      a.kc = const_cast<bf16*>(ptr(l, 16)); a.vc = const_cast<bf16*>(ptr(l, 17));
      a.n_kv = nkv; a.group = nq / nkv;
      a.scale_log2 = scale * 1.4426950408889634f;
      a.window = dims[7];
      a.splits = dims[8];
      a.ws = static_cast<float*>(shares);
      a.count = static_cast<int*>(count);
      a.out = mix; a.ldo = nq * D;
      for (int s = 0; s < M; ++s) { a.base[s] = base[s]; a.have[s] = have[s]; }
      if (D == 128) rc = a.group <= 8 ? launch_dec_attn<128, 8>(a, M, st) : launch_dec_attn<128, 16>(a, M, st);
      else rc = a.group <= 8 ? launch_dec_attn<64, 8>(a, M, st) : launch_dec_attn<64, 16>(a, M, st);
      if (rc != 0) return rc;
    }
    SkinnyParams o{};
    o.w[0] = ptr(l, 11);
    o.bias[0] = lt[l] == 2 ? nullptr : ptr(l, 19);
    for (int s = 0; s < kSkSegs; ++s) o.seg_end[s] = H;
    o.M = M; o.N = H; o.K = mix_n; o.ldw = mix_n;
    o.x = mix; o.ldx = mix_n;
    o.res = r; o.ldres = H;
    if ((rc = skinny<SK_RESID>(o, st)) != 0) return rc;
    SkinnyParams u{};
    if ((rc = input(u, ptr(l, 12))) != 0) return rc;
    u.w[0] = ptr(l, 13); u.w[1] = ptr(l, 14);
    u.N = I;
    u.y = mlp; u.ldy = I;
    if ((rc = skinny<SK_SWIGLU>(u, st)) != 0) return rc;
    SkinnyParams d{};
    d.w[0] = ptr(l, 15);
    for (int s = 0; s < kSkSegs; ++s) d.seg_end[s] = H;
    d.M = M; d.N = H; d.K = I; d.ldw = I;
    d.x = mlp; d.ldx = I;
    d.res = r; d.ldres = H;
    if ((rc = skinny<SK_RESID>(d, st)) != 0) return rc;
  }
  return row_norm(r, static_cast<const bf16*>(final_norm), static_cast<bf16*>(hidden), M, H, eps, norm_off, st);
}

}  // extern "C"
