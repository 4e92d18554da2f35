// In-chunk algebra of the chunked gated delta rule, forward and backward, one CTA per (chunk of 64 tokens, head).
//
// With unit keys / scaled unit queries k, q (L2-normalised here), write strengths b, cumulated log decays G inside the
// chunk, D_ij = exp(G_i - G_j) and A = strictly-lower(b_i k_i . k_j D_ij):
//
//     T = (I + A)^-1     u = T (b v)     w = T (b e^G k)     q~ = q e^G     k~ = k e^(G_last - G)
//     gamma = e^G_last   attn = lower(q k^T D)                            (chunk_fwd_kernel)
//     out = o_state + attn v_new                                          (chunk_out_kernel)
//
// feed the chunk-to-chunk recurrence of gdn_scan.cu; the backward kernels return the gradients of the packed rows.
//
// All sums are fp32 FMAs on fp32 operands.  As separate framework operations these terms took about forty launches that
// each moved [H, chunks, 64, 128] or [H, chunks, 64, 64] fp32 tensors (134 - 268 MB at 32 heads x 16384 tokens), among
// them a batched triangular solve that used a fraction of the chip.  Here a chunk is read once in the stream's own dtype
// through the row map (no padded copy), stays in shared memory, and only what the recurrence or the backward pass reads
// again is written.  What bounds the kernels then is the fp32 pipe (a 64 x 64 x 128 product is 4096 cycles of an SM)
// and the barriers between the phases; about 100 KB of shared memory keep two CTAs per SM so that one's barriers hide
// behind the other's products.
// One layer of 32 heads x 16384 tokens, forward + backward: 19.6 ms of device time as framework operations; here 1.26 (forward)
// + 0.27 (output) + 0.62 (output backward) + 2.14 (backward) ms.
//
// Role in the reference: the in-chunk Triton kernels of the FLA package behind `chunk_gated_delta_rule`
// (src/lmms_engine/models/qwen3_5/qwen3_5_ops.py:138-298).
#include "common.cuh"

namespace b200 {

using bf16 = __nv_bfloat16;
constexpr int CC = 64;            // tokens per chunk
constexpr int CD = 128;           // head dim of keys and values
constexpr int LB = CD + 4;        // row stride of [64, 128] buffers: 16-byte rows on distinct bank groups
constexpr int LS = CC + 4;        // row stride of [64, 64] buffers
constexpr int CT = 256;           // threads

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ float4 row4(const float* p) { return ld4(p); }
__device__ __forceinline__ float4 row4(const bf16* p) {
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y);
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void put4(float* p, const float4& v) { st4(p, v); }
__device__ __forceinline__ void put4(bf16* p, const float4& v) {
  *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b) { return a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w; }
__device__ __forceinline__ float sum16(float v) {  // over the sixteen lanes that share a row tile
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void fma4(float4& c, float a, const float4& b) {
  c.x = fmaf(a, b.x, c.x); c.y = fmaf(a, b.y, c.y); c.z = fmaf(a, b.z, c.z); c.w = fmaf(a, b.w, c.w);
}
__device__ __forceinline__ float4 scaled(const float4& a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }

// A thread of a [64, 128] result owns rows 4 ty .. 4 ty + 3 and columns 4 tx .. + 3 and 64 + 4 tx .. + 3.
struct Tile { float4 v[4][2]; };
__device__ __forceinline__ void zero(Tile& t) {
#pragma unroll
  for (int a = 0; a < 4; ++a) t.v[a][0] = t.v[a][1] = make_float4(0.f, 0.f, 0.f, 0.f);
}
// c[i] += sum over j < hi of L[i][j] R[j]          (L [64][LS], R [64][LB]; hi a multiple of four)
__device__ __forceinline__ void mul_rows(Tile& c, const float* L, const float* R, int ty, int tx, int hi) {
#pragma unroll 2
  for (int j = 0; j < hi; j += 4) {
    float4 l[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) l[a] = ld4(L + (4 * ty + a) * LS + j);
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) {
      const float4 r0 = ld4(R + (j + jj) * LB + 4 * tx), r1 = ld4(R + (j + jj) * LB + 64 + 4 * tx);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float s = jj == 0 ? l[a].x : jj == 1 ? l[a].y : jj == 2 ? l[a].z : l[a].w;
        fma4(c.v[a][0], s, r0);
        fma4(c.v[a][1], s, r1);
      }
    }
  }
}
// c[j] += sum over i >= lo of L[i][j] R[i]
__device__ __forceinline__ void mul_cols(Tile& c, const float* L, const float* R, int ty, int tx, int lo) {
#pragma unroll 4
  for (int i = lo; i < CC; ++i) {
    const float4 l = ld4(L + i * LS + 4 * ty);
    const float4 r0 = ld4(R + i * LB + 4 * tx), r1 = ld4(R + i * LB + 64 + 4 * tx);
    fma4(c.v[0][0], l.x, r0); fma4(c.v[0][1], l.x, r1);
    fma4(c.v[1][0], l.y, r0); fma4(c.v[1][1], l.y, r1);
    fma4(c.v[2][0], l.z, r0); fma4(c.v[2][1], l.z, r1);
    fma4(c.v[3][0], l.w, r0); fma4(c.v[3][1], l.w, r1);
  }
}
// acc[a][b] += X[ty + 16 a] . Y[tx + 16 b]: the threads of a quarter warp read consecutive rows of Y
__device__ __forceinline__ void mul_nt(float (&acc)[4][4], const float* X, const float* Y, int ty, int tx) {
#pragma unroll 2
  for (int d = 0; d < CD; d += 4) {
    float4 x[4], y[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) { x[a] = ld4(X + (ty + 16 * a) * LB + d); y[a] = ld4(Y + (tx + 16 * a) * LB + d); }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        acc[a][b] = fmaf(x[a].x, y[b].x, acc[a][b]);
        acc[a][b] = fmaf(x[a].y, y[b].y, acc[a][b]);
        acc[a][b] = fmaf(x[a].z, y[b].z, acc[a][b]);
        acc[a][b] = fmaf(x[a].w, y[b].w, acc[a][b]);
      }
  }
}
__device__ __forceinline__ void load_big(float* dst, const float* src) {  // contiguous [64, 128]
  for (int i = threadIdx.x; i < CC * CD / 4; i += CT) st4(dst + (i >> 5) * LB + (i & 31) * 4, ld4(src + i * 4));
}
__device__ __forceinline__ void load_small(float* dst, const float* src) {  // contiguous [64, 64]
  for (int i = threadIdx.x; i < CC * CC / 4; i += CT) st4(dst + (i >> 4) * LS + (i & 15) * 4, ld4(src + i * 4));
}
__device__ __forceinline__ void store_tile(float* dst, const Tile& t, int ty, int tx, int ld) {
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    st4(dst + (4 * ty + a) * ld + 4 * tx, t.v[a][0]);
    st4(dst + (4 * ty + a) * ld + 64 + 4 * tx, t.v[a][1]);
  }
}

template <typename T>
struct ChunkStream {           // packed rows of the documents: q, k, v [rows, H, 128] with row strides, g, beta [rows, H]
  const T *q, *k, *v;
  long ldq, ldk, ldv;
  const float *g, *beta;
  const int64_t* src;          // [n * 64] stream row of every chunk row; anything outside [0, rows) is a zero row
  long rows;
  int H, n;
  float scale;                 // of the unit queries
};
__device__ __forceinline__ long chunk_row(const int64_t* src, long rows, int chunk, int r) {
  const int64_t t = src[static_cast<long>(chunk) * CC + r];
  return (t >= 0 && t < rows) ? static_cast<long>(t) : -1;
}

// L2-normalised rows into `dst` (times `scale`), one warp per row; `rs` receives the inverse norms.
template <typename T>
__device__ __forceinline__ void load_unit(float* dst, float* rs, const T* x, long ld, const long* rowmap, int h, float scale) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int r = warp; r < CC; r += CT / 32) {
    const long row = rowmap[r];
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= 0) v = row4(x + row * ld + static_cast<long>(h) * CD + lane * 4);
    const float inv = rsqrtf(warp_sum(dot4(v, v)) + 1e-6f);
    if (lane == 0) rs[r] = inv;
    st4(dst + r * LB + lane * 4, scaled(scaled(v, inv), scale));
  }
}
// A cumulated log decay as the unevaluated sum of two floats.  Decays are exponentials of differences of these sums, so the error
// of a sum in 32 bits (2^-24 of its size, which is many times the difference) shows in every one of them; a scan over lanes
// rounds neighbours independently, which left the outputs 1.3 times as far from the exact rule as a sum in order (2.0e-6 against
// 1.5e-6 of the 2-norm at decays of up to 16; 2.2e-7 this way).
struct LogDecay {
  float hi, lo;
  __device__ __forceinline__ float minus(const LogDecay& o) const { return (hi - o.hi) + (lo - o.lo); }
};

// Cumulated log decays (summed in 64 bits) and write strengths of a chunk; ends with a barrier.
template <typename T>
__device__ __forceinline__ void load_gates(const ChunkStream<T>& p, long* rowmap, LogDecay* sG, float* sB, int chunk, int h) {
  __shared__ double first_half;
  const int tid = threadIdx.x, lane = tid & 31;
  double gv = 0.0;
  if (tid < CC) {
    const long row = chunk_row(p.src, p.rows, chunk, tid);
    rowmap[tid] = row;
    gv = row >= 0 ? static_cast<double>(p.g[row * p.H + h]) : 0.0;
    sB[tid] = row >= 0 ? p.beta[row * p.H + h] : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, gv, o);
      if (lane >= o) gv += up;
    }
    if (tid == 31) first_half = gv;
  }
  __syncthreads();
  if (tid < CC) {
    if (tid >= 32) gv += first_half;
    const float hi = static_cast<float>(gv);
    sG[tid] = {hi, fabsf(hi) < INFINITY ? static_cast<float>(gv - hi) : 0.f};
  }
  __syncthreads();
}

// T = (I + A)^-1 for strictly lower A: the four 16 x 16 diagonal blocks by substitution, then -T22 A21 T11 for blocks of
// 16 and 32; the upper blocks of T hold the intermediate products and are cleared again.  Ends with a barrier.
__device__ __forceinline__ void invert_unit_lower(const float* A, float* Tm) {
  const int tid = threadIdx.x;
  if (tid < CC) {
    const int b = tid & ~15, c = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float s = i == c ? 1.f : 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) s = fmaf(-A[(b + i) * LS + b + j], x[j], s);
      x[i] = s;
      Tm[(b + i) * LS + b + c] = s;
    }
  }
  __syncthreads();
#pragma unroll
  for (int m = 16; m <= 32; m *= 2) {
    const int blocks = CC / (2 * m), per = m * m;
    for (int e = tid; e < blocks * per; e += CT) {
      const int p = e / per, r = (e % per) / m, c = e % m, o = p * 2 * m;
      float s = 0.f;
      for (int j = c & ~3; j < m; ++j) s = fmaf(A[(o + m + r) * LS + o + j], Tm[(o + j) * LS + o + c], s);
      Tm[(o + r) * LS + o + m + c] = s;
    }
    __syncthreads();
    for (int e = tid; e < blocks * per; e += CT) {
      const int p = e / per, r = (e % per) / m, c = e % m, o = p * 2 * m;
      float s = 0.f;
      for (int j = 0; j <= r; ++j) s = fmaf(Tm[(o + m + r) * LS + o + m + j], Tm[(o + j) * LS + o + m + c], s);
      Tm[(o + m + r) * LS + o + c] = -s;
    }
    __syncthreads();
    // the next level and the products read entries above the diagonal (j in [c & ~3, c)): they have to be zero
    for (int e = tid; e < blocks * per; e += CT) {
      const int p = e / per, r = (e % per) / m, c = e % m, o = p * 2 * m;
      Tm[(o + r) * LS + o + m + c] = 0.f;
    }
    __syncthreads();
  }
}

constexpr int kFwdFloats = 2 * CC * LB + 2 * CC * LS;

template <typename T>
__global__ void __launch_bounds__(CT, 2)
chunk_fwd_kernel(const ChunkStream<T> p, float* __restrict__ w, float* __restrict__ u, float* __restrict__ qt, float* __restrict__ kt,
                 float* __restrict__ gamma, float* __restrict__ attn, float* __restrict__ Tinv, float* __restrict__ Amat) {
  extern __shared__ __align__(16) float sm[];
  float* sK = sm;
  float* sX = sK + CC * LB;      // queries, later values
  float* sA = sX + CC * LB;
  float* sT = sA + CC * LS;
  __shared__ LogDecay sG[CC];
  __shared__ float sB[CC], sE[CC], rs[CC];
  __shared__ long rowmap[CC];
  const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const long at = static_cast<long>(h) * p.n + chunk;
  load_gates(p, rowmap, sG, sB, chunk, h);
  load_unit(sK, rs, p.k, p.ldk, rowmap, h, 1.f);
  load_unit(sX, rs, p.q, p.ldq, rowmap, h, p.scale);
  const LogDecay g_last = sG[CC - 1];
  if (tid < CC) sE[tid] = expf(sG[tid].hi);
  if (tid == 0) gamma[at] = expf(g_last.hi);
  __syncthreads();
  for (int i = tid; i < CC * CD / 4; i += CT) {
    const int r = i >> 5, c = (i & 31) * 4;
    st4(qt + at * CC * CD + i * 4, scaled(ld4(sX + r * LB + c), sE[r]));
    st4(kt + at * CC * CD + i * 4, scaled(ld4(sK + r * LB + c), expf(g_last.minus(sG[r]))));
  }
  {
    float kk[4][4] = {}, qk[4][4] = {};
    mul_nt(kk, sK, sK, ty, tx);
    mul_nt(qk, sX, sK, ty, tx);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int i = ty + 16 * a, j = tx + 16 * b;
        const float d = i >= j ? expf(sG[i].minus(sG[j])) : 0.f;
        const float av = i > j ? kk[a][b] * sB[i] * d : 0.f;
        sA[i * LS + j] = av;
        sT[i * LS + j] = 0.f;
        Amat[at * CC * CC + i * CC + j] = av;
        attn[at * CC * CC + i * CC + j] = i >= j ? qk[a][b] * d : 0.f;
      }
  }
  __syncthreads();
  {  // values take the place of the queries
    const int warp = tid >> 5, lane = tid & 31;
    for (int r = warp; r < CC; r += CT / 32) {
      const long row = rowmap[r];
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row >= 0) v = row4(p.v + row * p.ldv + static_cast<long>(h) * CD + lane * 4);
      st4(sX + r * LB + lane * 4, v);
    }
  }
  invert_unit_lower(sA, sT);
  for (int i = tid; i < CC * CC / 4; i += CT) {
    const int r = i >> 4, c = (i & 15) * 4;
    float4 t = ld4(sT + r * LS + c);
    st4(Tinv + at * CC * CC + i * 4, t);
    t.x *= sB[c]; t.y *= sB[c + 1]; t.z *= sB[c + 2]; t.w *= sB[c + 3];
    st4(sT + r * LS + c, t);                                                      // T b
    t.x *= sE[c]; t.y *= sE[c + 1]; t.z *= sE[c + 2]; t.w *= sE[c + 3];
    st4(sA + r * LS + c, t);                                                      // T b e^G
  }
  __syncthreads();
  Tile t;
  zero(t);
  mul_rows(t, sT, sX, ty, tx, 4 * ty + 4);
  store_tile(u + at * CC * CD, t, ty, tx, CD);
  zero(t);
  mul_rows(t, sA, sK, ty, tx, 4 * ty + 4);
  store_tile(w + at * CC * CD, t, ty, tx, CD);
}

constexpr int kBwdFloats = 2 * CC * LB + 2 * CC * LS;

template <typename T>
__global__ void __launch_bounds__(CT, 2)
chunk_bwd_kernel(const ChunkStream<T> p, const float* __restrict__ w, const float* __restrict__ u, const float* __restrict__ attn,
                 const float* __restrict__ Tinv, const float* __restrict__ Amat, const float* __restrict__ dw,
                 const float* __restrict__ du, const float* __restrict__ dqt, const float* __restrict__ dkt,
                 const float* __restrict__ dgamma, const float* __restrict__ dattn, T* __restrict__ dq, T* __restrict__ dk,
                 T* __restrict__ dv, float* __restrict__ dg, float* __restrict__ dbeta) {
  extern __shared__ __align__(16) float sm[];
  float* B0 = sm;
  float* B1 = B0 + CC * LB;
  float* s0 = B1 + CC * LB;
  float* s1 = s0 + CC * LS;
  __shared__ LogDecay sG[CC];
  __shared__ float sB[CC], sE[CC], rq[CC], rk[CC], row_g[CC], row_t[CC], row_b[CC], col_e[CT / 32][CC];
  __shared__ long rowmap[CC];
  const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const long at = static_cast<long>(h) * p.n + chunk;
  const long big = at * CC * CD, small = at * CC * CC;
  const long ldo = static_cast<long>(p.H) * CD;   // gradients of the stream are dense [rows, H, 128]
  load_gates(p, rowmap, sG, sB, chunk, h);
  if (tid < CC) sE[tid] = expf(sG[tid].hi);
  load_small(s0, Tinv + small);
  load_big(B0, du + big);
  __syncthreads();
  const LogDecay g_last = sG[CC - 1];

  // d(b v) = T^T du, d(b e^G k) = T^T dw, dA = -(d(b v) u^T + d(b e^G k) w^T)
  float dA[4][4] = {};
  float db[4];
  Tile t;
  zero(t);
  mul_cols(t, s0, B0, ty, tx, 4 * ty);
  __syncthreads();
  store_tile(B1, t, ty, tx, LB);
  load_big(B0, u + big);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = 4 * ty + a;
    const long row = rowmap[r];
    float s = 0.f;
    if (row >= 0) {
      const T* vr = p.v + row * p.ldv + static_cast<long>(h) * CD + 4 * tx;
      s = dot4(t.v[a][0], row4(vr)) + dot4(t.v[a][1], row4(vr + 64));
      T* o = dv + row * ldo + static_cast<long>(h) * CD + 4 * tx;
      put4(o, scaled(t.v[a][0], sB[r]));
      put4(o + 64, scaled(t.v[a][1], sB[r]));
    }
    db[a] = sum16(s);
  }
  __syncthreads();
  mul_nt(dA, B1, B0, ty, tx);
  __syncthreads();
  load_big(B0, dw + big);
  __syncthreads();
  Tile dkb;   // first d(b e^G k), then d(b k)
  zero(dkb);
  mul_cols(dkb, s0, B0, ty, tx, 4 * ty);
  __syncthreads();
  store_tile(B1, dkb, ty, tx, LB);
  load_big(B0, w + big);
  __syncthreads();
  mul_nt(dA, B1, B0, ty, tx);

  // M = dA D, N = dattn D; dG from the decays: row sums minus column sums of dA A + dattn attn
  {
    float col[4] = {};
    const int warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const int i = ty + 16 * a;
      float rsum = 0.f;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int j = tx + 16 * b;
        float m = 0.f, nn = 0.f, e = 0.f;
        if (i >= j) {
          const float d = expf(sG[i].minus(sG[j]));
          const float da = dattn[small + i * CC + j];
          nn = da * d;
          e = da * attn[small + i * CC + j];
          if (i > j) {
            m = -dA[a][b] * d;
            e -= dA[a][b] * Amat[small + i * CC + j];
          }
        }
        s0[i * LS + j] = m;
        s1[i * LS + j] = nn;
        rsum += e;
        col[b] += e;
      }
      rsum = sum16(rsum);
      if (tx == 0) row_g[i] = rsum;
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const float c = col[b] + __shfl_xor_sync(0xffffffffu, col[b], 16);
      if (lane < 16) col_e[warp][tx + 16 * b] = c;
    }
  }
  __syncthreads();
  load_unit(B0, rk, p.k, p.ldk, rowmap, h, 1.f);
  load_unit(B1, rq, p.q, p.ldq, rowmap, h, p.scale);
  __syncthreads();

  float gsum[4];
  // queries: dq = dq~ e^G + N k
  zero(t);
  mul_rows(t, s1, B0, ty, tx, 4 * ty + 4);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = 4 * ty + a;
    const long row = rowmap[r];
    float gs = 0.f, qd = 0.f;
    float4 qh[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      qh[c] = ld4(B1 + r * LB + 64 * c + 4 * tx);
      const float4 kh = ld4(B0 + r * LB + 64 * c + 4 * tx);
      const float4 d = scaled(ld4(dqt + big + r * CD + 64 * c + 4 * tx), sE[r]);
      gs += dot4(d, qh[c]);
      gs += dot4(dkb.v[a][c], kh) * (sB[r] * sE[r]);      // d(b e^G k) . b e^G k
      fma4(t.v[a][c], 1.f, d);
      qd += dot4(t.v[a][c], qh[c]);
      dkb.v[a][c] = scaled(dkb.v[a][c], sE[r]);
    }
    gsum[a] = sum16(gs);
    qd = sum16(qd);
    if (row >= 0) {
      // q^ = scale q r: dq = scale r dq^ - (r / scale) q^ (q^ . dq^)
      const float f0 = p.scale * rq[r], f1 = -rq[r] / p.scale * qd;
      T* o = dq + row * ldo + static_cast<long>(h) * CD + 4 * tx;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float4 v = scaled(t.v[a][c], f0);
        fma4(v, f1, qh[c]);
        put4(o + 64 * c, v);
      }
    }
  }
  // keys
  mul_rows(dkb, s0, B0, ty, tx, 4 * ty + 4);              // d(b k) += M k
  zero(t);
  mul_cols(t, s1, B1, ty, tx, 4 * ty);                    // N^T q
  __syncthreads();
  for (int i = tid; i < CC * CC / 4; i += CT) {           // rows of M times b
    const int r = i >> 4;
    float* m = s0 + r * LS + (i & 15) * 4;
    st4(m, scaled(ld4(m), sB[r]));
  }
  __syncthreads();
  mul_cols(t, s0, B0, ty, tx, 4 * ty);                    // M^T b k
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const int r = 4 * ty + a;
    const long row = rowmap[r];
    const float fall = expf(g_last.minus(sG[r]));
    float ts = 0.f, bs = 0.f, kd = 0.f;
    float4 kh[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      kh[c] = ld4(B0 + r * LB + 64 * c + 4 * tx);
      const float4 d = scaled(ld4(dkt + big + r * CD + 64 * c + 4 * tx), fall);
      ts += dot4(d, kh[c]);
      bs += dot4(dkb.v[a][c], kh[c]);
      fma4(t.v[a][c], 1.f, d);
      fma4(t.v[a][c], sB[r], dkb.v[a][c]);
      kd += dot4(t.v[a][c], kh[c]);
    }
    ts = sum16(ts);
    bs = sum16(bs);
    kd = sum16(kd);
    if (row >= 0) {
      T* o = dk + row * ldo + static_cast<long>(h) * CD + 4 * tx;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        float4 v = t.v[a][c];
        fma4(v, -kd, kh[c]);
        put4(o + 64 * c, scaled(v, rk[r]));
      }
    }
    if (tx == 0) {
      row_t[r] = ts;
      row_b[r] = bs + db[a];
      row_g[r] += gsum[a] - ts;   // its row sum was written several barriers ago
    }
  }
  __syncthreads();
  if (tid < 32) {
    // dG of the rows (lane and lane + 32), the last one collecting k~ and gamma, then the reverse cumulated sum
    float lo = row_g[tid], hi = row_g[tid + 32];
#pragma unroll
    for (int wv = 0; wv < CT / 32; ++wv) { lo -= col_e[wv][tid]; hi -= col_e[wv][tid + 32]; }
    const float last = warp_sum(row_t[tid] + row_t[tid + 32]) + dgamma[at] * expf(g_last.hi);
    if (tid == 31) hi += last;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float dl = __shfl_down_sync(0xffffffffu, lo, o), dh = __shfl_down_sync(0xffffffffu, hi, o);
      if (tid + o < 32) { lo += dl; hi += dh; }
    }
    lo += __shfl_sync(0xffffffffu, hi, 0);
    const long r0 = rowmap[tid], r1 = rowmap[tid + 32];
    if (r0 >= 0) { dg[r0 * p.H + h] = lo; dbeta[r0 * p.H + h] = row_b[tid]; }
    if (r1 >= 0) { dg[r1 * p.H + h] = hi; dbeta[r1 * p.H + h] = row_b[tid + 32]; }
  }
}

// out[stream row] = o_state + attn v_new
constexpr int kOutFloats = CC * LB + CC * LS;
template <typename T>
__global__ void __launch_bounds__(CT)
chunk_out_kernel(const float* __restrict__ o_state, const float* __restrict__ attn, const float* __restrict__ vnew,
                 const int64_t* __restrict__ src, T* __restrict__ out, long rows, int H, int n) {
  extern __shared__ __align__(16) float sm[];
  float* sV = sm;
  float* sA = sV + CC * LB;
  const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const long at = static_cast<long>(h) * n + chunk;
  load_big(sV, vnew + at * CC * CD);
  load_small(sA, attn + at * CC * CC);
  Tile t;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 2; ++c) t.v[a][c] = ld4(o_state + at * CC * CD + (4 * ty + a) * CD + 64 * c + 4 * tx);
  __syncthreads();
  mul_rows(t, sA, sV, ty, tx, 4 * ty + 4);
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const long row = chunk_row(src, rows, chunk, 4 * ty + a);
    if (row < 0) continue;
    T* o = out + (row * H + h) * CD + 4 * tx;
    put4(o, t.v[a][0]);
    put4(o + 64, t.v[a][1]);
  }
}

// d o_state = dout (chunk layout), d v_new = attn^T dout, d attn = lower(dout v_new^T)
constexpr int kOutBwdFloats = 2 * CC * LB + CC * LS;
template <typename T>
__global__ void __launch_bounds__(CT, 2)
chunk_out_bwd_kernel(const T* __restrict__ dout, const float* __restrict__ attn, const float* __restrict__ vnew,
                     const int64_t* __restrict__ src, float* __restrict__ d_o, float* __restrict__ d_vnew,
                     float* __restrict__ d_attn, long rows, int H, int n) {
  extern __shared__ __align__(16) float sm[];
  float* sO = sm;
  float* sV = sO + CC * LB;
  float* sA = sV + CC * LB;
  const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const long at = static_cast<long>(h) * n + chunk;
  load_big(sV, vnew + at * CC * CD);
  load_small(sA, attn + at * CC * CC);
  for (int r = tid >> 5; r < CC; r += CT / 32) {
    const int c = (tid & 31) * 4;
    const long row = chunk_row(src, rows, chunk, r);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row >= 0) v = row4(dout + (row * H + h) * CD + c);
    st4(sO + r * LB + c, v);
    st4(d_o + at * CC * CD + r * CD + c, v);
  }
  __syncthreads();
  Tile t;
  zero(t);
  mul_cols(t, sA, sO, ty, tx, 4 * ty);
  store_tile(d_vnew + at * CC * CD, t, ty, tx, CD);
  float acc[4][4] = {};
  mul_nt(acc, sO, sV, ty, tx);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int i = ty + 16 * a, j = tx + 16 * b;
      d_attn[at * CC * CC + i * CC + j] = i >= j ? acc[a][b] : 0.f;
    }
}

template <typename K>
static int allow(K kernel, int floats) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, floats * 4) == cudaSuccess ? 0 : -3;
}

struct StreamArgs {
  const void *q, *k, *v;
  long ldq, ldk, ldv;
  const void *g, *beta, *src;
  long rows;
  int H, n;
  float scale;
};
template <typename T>
static ChunkStream<T> stream_of(const StreamArgs& a) {
  return {static_cast<const T*>(a.q), static_cast<const T*>(a.k), static_cast<const T*>(a.v), a.ldq, a.ldk, a.ldv,
          static_cast<const float*>(a.g), static_cast<const float*>(a.beta), static_cast<const int64_t*>(a.src), a.rows, a.H, a.n, a.scale};
}

template <typename T>
static int run_fwd(const StreamArgs& a, float* w, float* u, float* qt, float* kt, float* gamma, float* attn, float* Tinv,
                   float* Amat, cudaStream_t st) {
  static const int ok = allow(chunk_fwd_kernel<T>, kFwdFloats);
  if (ok != 0) return ok;
  chunk_fwd_kernel<T><<<dim3(a.n, a.H), CT, kFwdFloats * 4, st>>>(stream_of<T>(a), w, u, qt, kt, gamma, attn, Tinv, Amat);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // namespace b200

using namespace b200;
#define F(x) static_cast<const float*>(x)
#define FM(x) static_cast<float*>(x)

extern "C" {

// q, k, v: [rows, H, 128] with unit element stride, head stride 128 and row strides ldq / ldk / ldv (multiples of four),
// 16-byte aligned, bf16 (is_bf16) or fp32.  g, beta [rows, H] fp32 contiguous.  src [n * 64] int64.  Everything else fp32:
// w, u, qt, kt [H, n, 64, 128], attn, Tinv, Amat [H, n, 64, 64], gamma [H, n].
int b200_gdn_chunk_fwd(const void* q, const void* k, const void* v, long ldq, long ldk, long ldv, const void* g,
                       const void* beta, const void* src, long rows, int H, int n, float scale, int is_bf16, void* w, void* u,
                       void* qt, void* kt, void* gamma, void* attn, void* Tinv, void* Amat, cudaStream_t st) {
  if (H <= 0 || n <= 0) return 0;
  if ((ldq | ldk | ldv) & 3 || H > 65535) return -10;
  const StreamArgs a{q, k, v, ldq, ldk, ldv, g, beta, src, rows, H, n, scale};
  if (is_bf16) return run_fwd<bf16>(a, FM(w), FM(u), FM(qt), FM(kt), FM(gamma), FM(attn), FM(Tinv), FM(Amat), st);
  return run_fwd<float>(a, FM(w), FM(u), FM(qt), FM(kt), FM(gamma), FM(attn), FM(Tinv), FM(Amat), st);
}

// dq, dk, dv [rows, H, 128] in the stream's dtype and dg, dbeta [rows, H] fp32, contiguous: only rows that `src` names are
// written.
int b200_gdn_chunk_bwd(const void* q, const void* k, const void* v, long ldq, long ldk, long ldv, const void* g,
                       const void* beta, const void* src, long rows, int H, int n, float scale, int is_bf16, const void* w,
                       const void* u, const void* attn, const void* Tinv, const void* Amat, const void* dw, const void* du,
                       const void* dqt, const void* dkt, const void* dgamma, const void* dattn, void* dq, void* dk, void* dv,
                       void* dg, void* dbeta, cudaStream_t st) {
  if (H <= 0 || n <= 0) return 0;
  if ((ldq | ldk | ldv) & 3 || H > 65535) return -10;
  const StreamArgs a{q, k, v, ldq, ldk, ldv, g, beta, src, rows, H, n, scale};
  if (is_bf16) {
    static const int ok = allow(chunk_bwd_kernel<bf16>, kBwdFloats);
    if (ok != 0) return ok;
    chunk_bwd_kernel<bf16><<<dim3(n, H), CT, kBwdFloats * 4, st>>>(stream_of<bf16>(a), F(w), F(u), F(attn), F(Tinv), F(Amat), F(dw), F(du),
        F(dqt), F(dkt), F(dgamma), F(dattn), static_cast<bf16*>(dq), static_cast<bf16*>(dk), static_cast<bf16*>(dv), FM(dg), FM(dbeta));
  } else {
    static const int ok = allow(chunk_bwd_kernel<float>, kBwdFloats);
    if (ok != 0) return ok;
    chunk_bwd_kernel<float><<<dim3(n, H), CT, kBwdFloats * 4, st>>>(stream_of<float>(a), F(w), F(u), F(attn), F(Tinv), F(Amat), F(dw), F(du),
        F(dqt), F(dkt), F(dgamma), F(dattn), FM(dq), FM(dk), FM(dv), FM(dg), FM(dbeta));
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// out [rows, H, 128] contiguous, bf16 or fp32: rows that `src` names are written.
int b200_gdn_chunk_out(const void* o_state, const void* attn, const void* vnew, const void* src, void* out, long rows, int H, int n,
                       int is_bf16, cudaStream_t st) {
  if (H <= 0 || n <= 0) return 0;
  if (H > 65535) return -10;
  const int64_t* s = static_cast<const int64_t*>(src);
  if (is_bf16) {
    static const int ok = allow(chunk_out_kernel<bf16>, kOutFloats);
    if (ok != 0) return ok;
    chunk_out_kernel<bf16><<<dim3(n, H), CT, kOutFloats * 4, st>>>(F(o_state), F(attn), F(vnew), s, static_cast<bf16*>(out), rows, H, n);
  } else {
    static const int ok = allow(chunk_out_kernel<float>, kOutFloats);
    if (ok != 0) return ok;
    chunk_out_kernel<float><<<dim3(n, H), CT, kOutFloats * 4, st>>>(F(o_state), F(attn), F(vnew), s, FM(out), rows, H, n);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

int b200_gdn_chunk_out_bwd(const void* dout, const void* attn, const void* vnew, const void* src, void* d_o, void* d_vnew, void* d_attn,
                           long rows, int H, int n, int is_bf16, cudaStream_t st) {
  if (H <= 0 || n <= 0) return 0;
  if (H > 65535) return -10;
  const int64_t* s = static_cast<const int64_t*>(src);
  if (is_bf16) {
    static const int ok = allow(chunk_out_bwd_kernel<bf16>, kOutBwdFloats);
    if (ok != 0) return ok;
    chunk_out_bwd_kernel<bf16><<<dim3(n, H), CT, kOutBwdFloats * 4, st>>>(static_cast<const bf16*>(dout), F(attn), F(vnew), s, FM(d_o),
                                                                         FM(d_vnew), FM(d_attn), rows, H, n);
  } else {
    static const int ok = allow(chunk_out_bwd_kernel<float>, kOutBwdFloats);
    if (ok != 0) return ok;
    chunk_out_bwd_kernel<float><<<dim3(n, H), CT, kOutBwdFloats * 4, st>>>(F(dout), F(attn), F(vnew), s, FM(d_o), FM(d_vnew), FM(d_attn),
                                                                          rows, H, n);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

}  // extern "C"
