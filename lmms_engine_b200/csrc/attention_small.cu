// Attention over packed documents of at most 64 tokens (the 8 x 8-patch windows of a vision tower), forward and backward.
//
// One CTA of four warps per (document, key head): the whole document sits in shared memory, scores stay in registers, and
// the backward pass produces dQ, dK and dV of a document in one visit.  These calls are bound by moving q, k, v, o and their
// gradients once: a 64-token document of one head is 40 - 64 KB for 1 - 4 MFLOP, below a microsecond of mma.sync work, and
// several CTAs per SM overlap one's loads with another's products.  The tcgen05 kernels (attention_sm100.cu,
// attention_bwd_sm100.cu) take one document per 128-row tile and one CTA per SM: half of each tile is empty and every document
// pays the set-up of barriers, tensor memory and pipelines that only long key ranges amortise.
// 366 windows x 16 heads of 80 (21.9k patches): forward 0.90 -> 0.058 ms, backward 2.1 -> 0.23 ms (q, k, v, o and the gradients
// at 6.65 TB/s: 0.034 and 0.07 ms).
//
// Counterpart in the reference: flash_attn_varlen_func on the window boundaries (src/lmms_engine/kernels/attention.py:20-51).
#include "common.cuh"

namespace b200 {

using bf16 = __nv_bfloat16;
constexpr int kDoc = 64;        // longest document
constexpr int kPLd = kDoc + 8;  // row stride of the probability tiles

struct SmallP {
  const bf16 *q, *k, *v, *o, *dout;
  bf16 *out, *dq, *dk, *dv;
  float* lse;                    // [Hq, Tq]
  const int *cu_q, *cu_k;
  int Tq, Tk, Hq, Hkv, D;
  long ldq, ldk, ldv, ldo, lddo, lddq, lddk, lddv;
  float scale, scale_log2;
  int causal, window_left;
  int* status;
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)) : "memory");
}
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void cp16(bf16* dst, const bf16* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Rows [start, start + len) of one head into [64][DP + 8]; rows past the document and columns past D are zero.
template <int DP>
__device__ __forceinline__ void load_rows(bf16* dst, const bf16* src, long ld, int start, int len, int head, int D) {
  constexpr int V = DP / 8;
  for (int i = threadIdx.x; i < kDoc * V; i += 128) {
    const int r = i / V, c = (i - r * V) * 8;
    bf16* d = dst + r * (DP + 8) + c;
    if (r < len && c < D) cp16(d, src + static_cast<long>(start + r) * ld + static_cast<long>(head) * D + c);
    else *reinterpret_cast<uint4*>(d) = make_uint4(0u, 0u, 0u, 0u);
  }
}
// acc[16 rows of this warp][64] = X rows . Y rows^T
template <int DP>
__device__ __forceinline__ void rows_dot(float (&acc)[8][4], const bf16* X, const bf16* Y, int warp, int lane) {
  constexpr int LD = DP + 8;
#pragma unroll
  for (int n = 0; n < 8; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
#pragma unroll
  for (int kk = 0; kk < DP / 16; ++kk) {
    uint32_t a[4];
    ldsm4(a, X + (warp * 16 + (lane & 15)) * LD + kk * 16 + (lane >> 4) * 8);
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      // two eight-key tiles: matrices (keys 0-7, k 0-7), (keys 0-7, k 8-15), (keys 8-15, k 0-7), (keys 8-15, k 8-15)
      uint32_t b[4];
      ldsm4(b, Y + (n * 16 + (lane & 7) + ((lane >> 4) << 3)) * LD + kk * 16 + ((lane >> 3) & 1) * 8);
      mma16816(acc[2 * n], a, b[0], b[1]);
      mma16816(acc[2 * n + 1], a, b[2], b[3]);
    }
  }
}
// acc[16][DP] += A (four 16-wide k steps of fragments) Y, Y [64][DP + 8]
template <int DP>
__device__ __forceinline__ void frags_times(float (&acc)[DP / 8][4], const uint32_t (&a)[4][4], const bf16* Y, int lane) {
  constexpr int LD = DP + 8;
#pragma unroll
  for (int kk = 0; kk < 4; ++kk)
#pragma unroll
    for (int n = 0; n < DP / 16; ++n) {
      uint32_t b[4];
      ldsm4_t(b, Y + (kk * 16 + (lane & 15)) * LD + n * 16 + (lane >> 4) * 8);
      mma16816(acc[2 * n], a[kk], b[0], b[1]);
      mma16816(acc[2 * n + 1], a[kk], b[2], b[3]);
    }
}
// 16 x DP accumulator of this warp -> its rows of a [64][DP + 8] buffer, as bf16
template <int DP>
__device__ __forceinline__ void stage(bf16* dst, const float (&acc)[DP / 8][4], float s0, float s1, int warp, int lane) {
  const int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int n = 0; n < DP / 8; ++n) {
    bf16* p = dst + (warp * 16 + g) * (DP + 8) + n * 8 + 2 * t;
    *reinterpret_cast<uint32_t*>(p) = pack_bf16x2(acc[n][0] * s0, acc[n][1] * s0);
    *reinterpret_cast<uint32_t*>(p + 8 * (DP + 8)) = pack_bf16x2(acc[n][2] * s1, acc[n][3] * s1);
  }
}
// this warp's 16 rows of a staged buffer -> global rows
template <int DP>
__device__ __forceinline__ void write_rows(bf16* dst, long ld, const bf16* src, int start, int len, int head, int D, int warp, int lane) {
  __syncwarp();
  const int V = D / 8;
  for (int i = lane; i < 16 * V; i += 32) {
    const int r = warp * 16 + i / V, c = (i % V) * 8;
    if (r < len)
      *reinterpret_cast<uint4*>(dst + static_cast<long>(start + r) * ld + static_cast<long>(head) * D + c) =
          *reinterpret_cast<const uint4*>(src + r * (DP + 8) + c);
  }
}
struct Doc {
  int q0, lq, k0, lk;
  __device__ __forceinline__ bool find(const SmallP& p, int d) {
    q0 = p.cu_q[d]; lq = p.cu_q[d + 1] - q0;
    k0 = p.cu_k[d]; lk = p.cu_k[d + 1] - k0;
    if (!doc_in_bounds(q0, lq, p.Tq, p.status) || !doc_in_bounds(k0, lk, p.Tk, p.status)) return false;
    if (lq > kDoc || lk > kDoc) {  // the caller promises documents of at most kDoc tokens
      if (p.status != nullptr) atomicExch(p.status, kStatusBadShape);
      return false;
    }
    return true;
  }
  // bottom-right aligned like the long-document kernels
  __device__ __forceinline__ bool sees(const SmallP& p, int qi, int kj) const {
    const int at = qi + lk - lq;
    return kj < lk && (!p.causal || kj <= at) && (p.window_left < 0 || kj >= at - p.window_left);
  }
};

template <int DP>
__global__ void __launch_bounds__(128) attn_small_fwd_kernel(const SmallP p) {
  extern __shared__ __align__(16) uint8_t dyn[];
  bf16* sQ = reinterpret_cast<bf16*>(dyn);
  bf16* sK = sQ + kDoc * (DP + 8);
  bf16* sV = sK + kDoc * (DP + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int head = blockIdx.x, kvh = head / (p.Hq / p.Hkv);
  Doc d;
  if (!d.find(p, blockIdx.y)) return;
  load_rows<DP>(sQ, p.q, p.ldq, d.q0, d.lq, head, p.D);
  load_rows<DP>(sK, p.k, p.ldk, d.k0, d.lk, kvh, p.D);
  load_rows<DP>(sV, p.v, p.ldv, d.k0, d.lk, kvh, p.D);
  cp_wait();
  __syncthreads();
  if (warp * 16 >= d.lq) return;
  float s[8][4];
  rows_dot<DP>(s, sQ, sK, warp, lane);
  float mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.f, 0.f};
#pragma unroll
  for (int n = 0; n < 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s[n][j] = d.sees(p, warp * 16 + g + 8 * (j >> 1), n * 8 + 2 * t + (j & 1)) ? s[n][j] * p.scale_log2 : -INFINITY;
      mx[j >> 1] = fmaxf(mx[j >> 1], s[n][j]);
    }
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
    mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
  }
  uint32_t pf[4][4];
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float m = mx[j >> 1] == -INFINITY ? 0.f : mx[j >> 1];
      e[j] = fast_exp2(s[n][j] - m);
      sum[j >> 1] += e[j];
    }
    pf[n >> 1][(n & 1) * 2] = pack_bf16x2(e[0], e[1]);
    pf[n >> 1][(n & 1) * 2 + 1] = pack_bf16x2(e[2], e[3]);
  }
  float inv[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 1);
    sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], 2);
    inv[r] = sum[r] > 0.f ? 1.f / sum[r] : 0.f;
    const int row = warp * 16 + g + 8 * r;
    if (t == 0 && row < d.lq)
      p.lse[static_cast<size_t>(head) * p.Tq + d.q0 + row] = sum[r] > 0.f ? (mx[r] + log2f(sum[r])) * 0.6931471805599453f : -INFINITY;
  }
  float o[DP / 8][4];
#pragma unroll
  for (int n = 0; n < DP / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
  frags_times<DP>(o, pf, sV, lane);
  __syncwarp();
  stage<DP>(sQ, o, inv[0], inv[1], warp, lane);   // only this warp reads these rows of sQ
  write_rows<DP>(p.out, p.ldo, sQ, d.q0, d.lq, head, p.D, warp, lane);
}

// The query heads of a group are visited one after the other and dK, dV stay in registers meanwhile.
template <int DP>
__global__ void __launch_bounds__(128) attn_small_bwd_kernel(const SmallP p) {
  extern __shared__ __align__(16) uint8_t dyn[];
  constexpr int LD = DP + 8;
  bf16* sK = reinterpret_cast<bf16*>(dyn);
  bf16* sV = sK + kDoc * LD;
  bf16* sQ = sV + kDoc * LD;
  bf16* sG = sQ + kDoc * LD;     // dO
  bf16* sP = sG + kDoc * LD;     // [64 queries][kPLd]
  bf16* sS = sP + kDoc * kPLd;   // dS
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int kvh = blockIdx.x, group = p.Hq / p.Hkv;
  Doc d;
  if (!d.find(p, blockIdx.y)) return;
  load_rows<DP>(sK, p.k, p.ldk, d.k0, d.lk, kvh, p.D);
  load_rows<DP>(sV, p.v, p.ldv, d.k0, d.lk, kvh, p.D);
  float dk[DP / 8][4], dv[DP / 8][4];
#pragma unroll
  for (int n = 0; n < DP / 8; ++n)
#pragma unroll
    for (int j = 0; j < 4; ++j) dk[n][j] = dv[n][j] = 0.f;
  for (int hg = 0; hg < group; ++hg) {
    const int head = kvh * group + hg;
    if (hg > 0) __syncthreads();
    load_rows<DP>(sQ, p.q, p.ldq, d.q0, d.lq, head, p.D);
    load_rows<DP>(sG, p.dout, p.lddo, d.q0, d.lq, head, p.D);
    cp_wait();
    __syncthreads();
    // delta and log-sum-exp of this thread's two rows; the four lanes of a row share the columns
    float delta[2] = {0.f, 0.f}, lse2[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = warp * 16 + g + 8 * r;
      lse2[r] = INFINITY;
      if (row < d.lq) {
        const bf16* orow = p.o + static_cast<long>(d.q0 + row) * p.ldo + static_cast<long>(head) * p.D;
        for (int c = t * 8; c < p.D; c += 32) {
          const uint4 a = *reinterpret_cast<const uint4*>(orow + c);
          const uint4 b = *reinterpret_cast<const uint4*>(sG + row * LD + c);
          const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 x = unpack_bf16x2(aw[j]), y = unpack_bf16x2(bw[j]);
            delta[r] += x.x * y.x + x.y * y.y;
          }
        }
        const float l = p.lse[static_cast<size_t>(head) * p.Tq + d.q0 + row];
        if (l > -INFINITY) lse2[r] = l * 1.4426950408889634f;
      }
      delta[r] += __shfl_xor_sync(0xffffffffu, delta[r], 1);
      delta[r] += __shfl_xor_sync(0xffffffffu, delta[r], 2);
    }
    uint32_t pf[4][4], sf[4][4];
    {
      float s[8][4], dp[8][4];
      rows_dot<DP>(s, sQ, sK, warp, lane);
      rows_dot<DP>(dp, sG, sV, warp, lane);
#pragma unroll
      for (int n = 0; n < 8; ++n) {
        float pv[4], ds[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool vis = d.sees(p, warp * 16 + g + 8 * (j >> 1), n * 8 + 2 * t + (j & 1));
          pv[j] = vis ? fast_exp2(fmaf(s[n][j], p.scale_log2, -lse2[j >> 1])) : 0.f;   // rows past the document: 2^-inf
          ds[j] = pv[j] * (dp[n][j] - delta[j >> 1]) * p.scale;
        }
        pf[n >> 1][(n & 1) * 2] = pack_bf16x2(pv[0], pv[1]);
        pf[n >> 1][(n & 1) * 2 + 1] = pack_bf16x2(pv[2], pv[3]);
        sf[n >> 1][(n & 1) * 2] = pack_bf16x2(ds[0], ds[1]);
        sf[n >> 1][(n & 1) * 2 + 1] = pack_bf16x2(ds[2], ds[3]);
        const int at = (warp * 16 + g) * kPLd + n * 8 + 2 * t;
        *reinterpret_cast<uint32_t*>(sP + at) = pf[n >> 1][(n & 1) * 2];
        *reinterpret_cast<uint32_t*>(sP + at + 8 * kPLd) = pf[n >> 1][(n & 1) * 2 + 1];
        *reinterpret_cast<uint32_t*>(sS + at) = sf[n >> 1][(n & 1) * 2];
        *reinterpret_cast<uint32_t*>(sS + at + 8 * kPLd) = sf[n >> 1][(n & 1) * 2 + 1];
      }
    }
    float dq[DP / 8][4];
#pragma unroll
    for (int n = 0; n < DP / 8; ++n) dq[n][0] = dq[n][1] = dq[n][2] = dq[n][3] = 0.f;
    frags_times<DP>(dq, sf, sK, lane);
    __syncthreads();   // P and dS of all queries are in place
    // keys of this warp: A = P^T / dS^T, read transposed
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      // matrices (queries 0-7, keys 0-7), (q 0-7, keys 8-15), (q 8-15, keys 0-7), (q 8-15, keys 8-15), each transposed
      const int at = (kk * 16 + (lane & 7) + ((lane >> 4) << 3)) * kPLd + warp * 16 + ((lane >> 3) & 1) * 8;
      ldsm4_t(pf[kk], sP + at);
      ldsm4_t(sf[kk], sS + at);
    }
    frags_times<DP>(dv, pf, sG, lane);
    frags_times<DP>(dk, sf, sQ, lane);
    __syncthreads();   // everybody is done with q and dO
    stage<DP>(sQ, dq, 1.f, 1.f, warp, lane);
    write_rows<DP>(p.dq, p.lddq, sQ, d.q0, d.lq, head, p.D, warp, lane);
  }
  __syncthreads();
  stage<DP>(sK, dk, 1.f, 1.f, warp, lane);
  stage<DP>(sV, dv, 1.f, 1.f, warp, lane);
  write_rows<DP>(p.dk, p.lddk, sK, d.k0, d.lk, kvh, p.D, warp, lane);
  write_rows<DP>(p.dv, p.lddv, sV, d.k0, d.lk, kvh, p.D, warp, lane);
}

// Head tiles of 64, 80 and 128: what a head does not fill is shared memory and products with zeros.  366 windows of 64 x 16 heads,
// forward / backward, us: heads of 80 59 / 235 on a tile of 80, 78 / 270 on one of 128 (heads of 72 60 / 233 and 78 / 262); heads
// of 64 47 / 199 on a tile of 64, 55 / 213 on one of 80.  Heads of 96 and 112 take 128: no configuration here has them.
template <int DP>
static int launch_fwd(const SmallP& p, int n_docs, cudaStream_t st) {
  constexpr int smem = 3 * kDoc * (DP + 8) * 2;
  static const cudaError_t e = cudaFuncSetAttribute(attn_small_fwd_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return -3;
  attn_small_fwd_kernel<DP><<<dim3(p.Hq, n_docs), 128, smem, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
template <int DP>
static int launch_bwd(const SmallP& p, int n_docs, cudaStream_t st) {
  constexpr int smem = (4 * kDoc * (DP + 8) + 2 * kDoc * kPLd) * 2;
  static const cudaError_t e = cudaFuncSetAttribute(attn_small_bwd_kernel<DP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return -3;
  attn_small_bwd_kernel<DP><<<dim3(p.Hkv, n_docs), 128, smem, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
static bool bad(const SmallP& p, int n_docs) {
  return p.D % 8 || p.D > 128 || p.D <= 0 || p.Hkv <= 0 || p.Hq % p.Hkv || n_docs > 65535 ||
         ((p.ldq | p.ldk | p.ldv | p.ldo | p.lddo | p.lddq | p.lddk | p.lddv) & 7);
}

}  // namespace b200

using namespace b200;

extern "C" {

// Documents of at most 64 queries and 64 keys; rows of contiguous heads at strides that are multiples of 8 elements, 16-byte
// aligned.  lse [Hq, Tq] fp32, natural logarithm.
int b200_attn_small_fwd(const void* q, const void* k, const void* v, void* o, void* lse, const void* cu_q, const void* cu_k,
                        int n_docs, int Tq, int Tk, int Hq, int Hkv, int D, long ldq, long ldk, long ldv, long ldo, float scale,
                        int causal, int window_left, int* status, cudaStream_t st) {
  if (n_docs <= 0 || Tq <= 0) return 0;
  SmallP p{};
  p.q = static_cast<const bf16*>(q); p.k = static_cast<const bf16*>(k); p.v = static_cast<const bf16*>(v);
  p.out = static_cast<bf16*>(o); p.lse = static_cast<float*>(lse);
  p.cu_q = static_cast<const int*>(cu_q); p.cu_k = static_cast<const int*>(cu_k);
  p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv; p.D = D;
  p.ldq = ldq; p.ldk = ldk; p.ldv = ldv; p.ldo = ldo;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal; p.window_left = window_left; p.status = status;
  if (bad(p, n_docs)) return -10;
  return D <= 64 ? launch_fwd<64>(p, n_docs, st) : D <= 80 ? launch_fwd<80>(p, n_docs, st) : launch_fwd<128>(p, n_docs, st);
}

int b200_attn_small_bwd(const void* q, const void* k, const void* v, const void* o, const void* dout, const void* lse, void* dq,
                        void* dk, void* dv, const void* cu_q, const void* cu_k, int n_docs, int Tq, int Tk, int Hq, int Hkv, int D,
                        long ldq, long ldk, long ldv, long ldo, long lddo, long lddq, long lddk, long lddv, float scale, int causal,
                        int window_left, int* status, cudaStream_t st) {
  if (n_docs <= 0 || Tq <= 0) return 0;
  SmallP p{};
  p.q = static_cast<const bf16*>(q); p.k = static_cast<const bf16*>(k); p.v = static_cast<const bf16*>(v);
  p.o = static_cast<const bf16*>(o); p.dout = static_cast<const bf16*>(dout);
  p.lse = const_cast<float*>(static_cast<const float*>(lse));
  p.dq = static_cast<bf16*>(dq); p.dk = static_cast<bf16*>(dk); p.dv = static_cast<bf16*>(dv);
  p.cu_q = static_cast<const int*>(cu_q); p.cu_k = static_cast<const int*>(cu_k);
  p.Tq = Tq; p.Tk = Tk; p.Hq = Hq; p.Hkv = Hkv; p.D = D;
  p.ldq = ldq; p.ldk = ldk; p.ldv = ldv; p.ldo = ldo; p.lddo = lddo; p.lddq = lddq; p.lddk = lddk; p.lddv = lddv;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f;
  p.causal = causal; p.window_left = window_left; p.status = status;
  if (bad(p, n_docs)) return -10;
  return D <= 64 ? launch_bwd<64>(p, n_docs, st) : D <= 80 ? launch_bwd<80>(p, n_docs, st) : launch_bwd<128>(p, n_docs, st);
}

}  // extern "C"
