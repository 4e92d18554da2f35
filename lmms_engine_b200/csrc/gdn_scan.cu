// Chunk-to-chunk part of the gated delta rule (Gated-DeltaNet linear attention), forward and backward.
//
// Per head the rule carries a state S [DK, dv] across chunks of C = 64 tokens:
//
//     v_new_i = u_i - w_i S_i          o_i = q~_i S_i          S_{i+1} = gamma_i S_i + k~_i^T v_new_i
//
// with S = 0 at the first chunk of every document (reset flag).  w, u (in-chunk corrected keys / values), q~ = q exp(g),
// k~ = k exp(g_last - g) and gamma = exp(g_last) come from gdn_chunk.cu.
//
// Only what the next state needs is sequential.  The scan kernels (one CTA per head and 32 columns of dv, state slice in shared
// memory for the whole sequence) therefore do two products per chunk forward (w S, k~^T v_new) and three backward (k~ dS, q~^T d_o,
// w^T d v_new) and write down the state (its gradient) at every chunk; o and the gradients of w, q~, k~ and gamma follow from
// those histories in kernels with one CTA per (chunk, head), which fill the chip and sum over all of dv at once.
// With everything in the scan, 128 CTAs did three and six products per chunk in sequence and the backward one wrote its three
// [64, 128] results once per dv slice (3.2 GB of partial sums a layer at 32 heads x 16384 tokens).
// One layer at that size, ms: forward scan 2.19 -> 1.46 + 0.67 (o), backward scan with its partial sums 5.5 + 0.75 -> 2.10 + 1.43.
// All products are fp32 FMAs.  What bounds the scans is the chain of barriers and products of 256 chunks, the others the fp32 pipe.
//
// Role in the reference: the `chunk_gated_delta_rule` Triton kernels of the FLA package used by
// src/lmms_engine/models/qwen3_5/qwen3_5_ops.py (gated delta net forward of the patched layers).
#include <cuda_runtime.h>

namespace b200 {

constexpr int DK = 128;   // key head dim
constexpr int C = 64;     // chunk length
constexpr int DVT = 32;   // dv columns per scan CTA
constexpr int LDK = DK + 4;   // padded rows: conflict-free column reads, 16-byte aligned float4 rows
constexpr int LDV = DVT + 4;
constexpr int THREADS = 256;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }

__device__ __forceinline__ void cp_async16(float* dst_smem, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst_smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// stage a [C, DK] fp32 block (contiguous in global memory) into padded shared memory with asynchronous 16-byte
// copies: the caller commits the group and waits for it before the block is read
__device__ __forceinline__ void stage_ck(float* dst, const float* __restrict__ src) {
  for (int idx = threadIdx.x; idx < C * DK / 4; idx += THREADS) {
    const int r = idx / (DK / 4), c4 = idx - r * (DK / 4);
    cp_async16(dst + r * LDK + c4 * 4, src + r * DK + c4 * 4);
  }
}
// stage the [C, DVT] slice of a [C, dv] block
__device__ __forceinline__ void stage_slice(float* dst, const float* __restrict__ src, int dv) {
  for (int idx = threadIdx.x; idx < C * DVT / 4; idx += THREADS) {
    const int r = idx / (DVT / 4), c4 = idx - r * (DVT / 4);
    cp_async16(dst + r * LDV + c4 * 4, src + static_cast<long>(r) * dv + c4 * 4);
  }
}

// [C, DVT] = A [C, DK] B [DK, DVT] with the key dimension split over the two halves of the CTA: a thread owns rows ty + 16 a and
// four columns, so that eight 16-byte reads feed 64 FMAs (two rows a thread over the whole dimension read more than they fed).
// The upper half parks its part in `park`; after the caller's barrier the lower half adds it.
__device__ __forceinline__ void rows_times_state(const float* A, const float* B, int half, int ty, int c0, float (&acc)[4][4]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 4; ++b) acc[a][b] = 0.f;
  const int k_lo = half * (DK / 2);
#pragma unroll 4
  for (int kk = k_lo; kk < k_lo + DK / 2; kk += 4) {
    float4 x[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) x[a] = ld4(A + (ty + 16 * a) * LDK + kk);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 b = ld4(B + (kk + j) * LDV + c0);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float s = j == 0 ? x[a].x : j == 1 ? x[a].y : j == 2 ? x[a].z : x[a].w;
        acc[a][0] += s * b.x; acc[a][1] += s * b.y; acc[a][2] += s * b.z; acc[a][3] += s * b.w;
      }
    }
  }
}

// acc[4][4] += sign * A[:, k0..k0+3]^T * V[:, c0..c0+3]   (A [C, DK] padded, V [C, DVT] padded)
__device__ __forceinline__ void transposed_times_rows(const float* A, const float* V, int k0, int c0, float sign,
                                                      float acc[4][4]) {
#pragma unroll 4
  for (int r = 0; r < C; ++r) {
    const float4 a = ld4(A + r * LDK + k0);
    float4 v = ld4(V + r * LDV + c0);
    v.x *= sign; v.y *= sign; v.z *= sign; v.w *= sign;
    acc[0][0] += a.x * v.x; acc[0][1] += a.x * v.y; acc[0][2] += a.x * v.z; acc[0][3] += a.x * v.w;
    acc[1][0] += a.y * v.x; acc[1][1] += a.y * v.y; acc[1][2] += a.y * v.z; acc[1][3] += a.y * v.w;
    acc[2][0] += a.z * v.x; acc[2][1] += a.z * v.y; acc[2][2] += a.z * v.z; acc[2][3] += a.z * v.w;
    acc[3][0] += a.w * v.x; acc[3][1] += a.w * v.y; acc[3][2] += a.w * v.z; acc[3][3] += a.w * v.w;
  }
}

constexpr int kScanFwdSmem = (2 * C * LDK + DK * LDV + 2 * C * LDV) * 4;

__global__ void __launch_bounds__(THREADS, 1)
gdn_scan_fwd_kernel(const float* __restrict__ w, const float* __restrict__ u, const float* __restrict__ kt,
                    const float* __restrict__ gamma, const int* __restrict__ reset, float* __restrict__ vnew,
                    float* __restrict__ hist, int n, int dv) {
  extern __shared__ __align__(16) float smem[];
  float* sW = smem;
  float* sK = sW + C * LDK;
  float* sS = sK + C * LDK;    // [DK][LDV]
  float* sV = sS + DK * LDV;   // [C][LDV]
  float* sX = sV + C * LDV;    // [C][LDV] the upper half's part of w S
  const int h = blockIdx.x, slice = blockIdx.y, tid = threadIdx.x;
  const int half = tid >> 7, ty = (tid & 127) >> 3, c0 = 4 * (tid & 7), k0 = 4 * (tid >> 3);
  const long col = static_cast<long>(slice) * DVT;
  for (int idx = tid; idx < DK * LDV; idx += THREADS) sS[idx] = 0.f;
  // the next chunk's w loads while the state update runs, the chunk's k~ while the product with the state runs
  stage_ck(sW, w + static_cast<long>(h) * n * C * DK);
  cp_async_commit();
  for (int i = 0; i < n; ++i) {
    const long chunk = static_cast<long>(h) * n + i, tok = chunk * C;
    if (reset[i]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) st4(sS + (k0 + j) * LDV + c0, make_float4(0.f, 0.f, 0.f, 0.f));
    }
    float4 uu[4];
    if (half == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) uu[a] = ld4(u + (tok + ty + 16 * a) * dv + col + c0);
    }
    const float g = gamma[chunk];
    cp_async_wait<0>();
    __syncthreads();   // w and the state are in place; nobody reads k~ or v_new of the chunk before any more
    stage_ck(sK, kt + chunk * C * DK);
    cp_async_commit();
    // state before this chunk
    float* hrow = hist + chunk * DK * dv + col;
#pragma unroll
    for (int j = 0; j < 4; ++j) st4(hrow + static_cast<long>(k0 + j) * dv + c0, ld4(sS + (k0 + j) * LDV + c0));
    float p[4][4];
    rows_times_state(sW, sS, half, ty, c0, p);
    if (half == 1) {
#pragma unroll
      for (int a = 0; a < 4; ++a) st4(sX + (ty + 16 * a) * LDV + c0, make_float4(p[a][0], p[a][1], p[a][2], p[a][3]));
    }
    __syncthreads();   // w has been read by everybody
    if (i + 1 < n) stage_ck(sW, w + (chunk + 1) * C * DK);
    cp_async_commit();
    if (half == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int r = ty + 16 * a;
        const float4 x = ld4(sX + r * LDV + c0);
        const float4 vn = make_float4(uu[a].x - (p[a][0] + x.x), uu[a].y - (p[a][1] + x.y), uu[a].z - (p[a][2] + x.z), uu[a].w - (p[a][3] + x.w));
        st4(vnew + (tok + r) * dv + col + c0, vn);
        st4(sV + r * LDV + c0, vn);
      }
    }
    cp_async_wait<1>();   // k~ (the next w may still be on its way)
    __syncthreads();
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 sv = ld4(sS + (k0 + j) * LDV + c0);   // own tile: only this thread rewrites it
      acc[j][0] = g * sv.x; acc[j][1] = g * sv.y; acc[j][2] = g * sv.z; acc[j][3] = g * sv.w;
    }
    transposed_times_rows(sK, sV, k0, c0, 1.f, acc);
#pragma unroll
    for (int j = 0; j < 4; ++j) st4(sS + (k0 + j) * LDV + c0, make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]));
    // the loop-top barrier orders these writes (and the reads of k~ / v_new) before the next chunk's use
  }
  cp_async_wait<0>();
}

constexpr int kScanBwdSmem = (3 * C * LDK + DK * LDV + 3 * C * LDV) * 4;

// du = total gradient of v_new; dhist = gradient of the state after every chunk.
__global__ void __launch_bounds__(THREADS, 1)
gdn_scan_bwd_kernel(const float* __restrict__ w, const float* __restrict__ qt, const float* __restrict__ kt,
                    const float* __restrict__ gamma, const int* __restrict__ reset, const float* __restrict__ d_vnew,
                    const float* __restrict__ d_o, float* __restrict__ du, float* __restrict__ dhist, int n, int dv) {
  extern __shared__ __align__(16) float smem[];
  float* sW = smem;
  float* sQ = sW + C * LDK;
  float* sK = sQ + C * LDK;
  float* sD = sK + C * LDK;    // [DK][LDV] gradient of the state after the chunk
  float* sO = sD + DK * LDV;   // [C][LDV] d_o
  float* sT = sO + C * LDV;    // [C][LDV] total gradient of v_new
  float* sX = sT + C * LDV;
  const int h = blockIdx.x, slice = blockIdx.y, tid = threadIdx.x;
  const int half = tid >> 7, ty = (tid & 127) >> 3, c0 = 4 * (tid & 7), k0 = 4 * (tid >> 3);
  const long col = static_cast<long>(slice) * DVT;
  for (int idx = tid; idx < DK * LDV; idx += THREADS) sD[idx] = 0.f;
  const long last = static_cast<long>(h) * n + n - 1;
  // k~ of the next chunk loads while the two updates run; w, q~ and d_o while the product with the state's gradient runs
  stage_ck(sK, kt + last * C * DK);
  cp_async_commit();
  for (int i = n - 1; i >= 0; --i) {
    const long chunk = static_cast<long>(h) * n + i, tok = chunk * C;
    float4 e[4];
    if (half == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) e[a] = ld4(d_vnew + (tok + ty + 16 * a) * dv + col + c0);
    }
    const float g = gamma[chunk];
    const bool cut = reset[i] != 0;
    cp_async_wait<0>();
    __syncthreads();   // k~ and dS are in place; nobody reads w, q~, d_o of the chunk before any more
    stage_ck(sW, w + chunk * C * DK);
    stage_ck(sQ, qt + chunk * C * DK);
    stage_slice(sO, d_o + tok * dv + col, dv);
    cp_async_commit();
    float* hrow = dhist + chunk * DK * dv + col;
#pragma unroll
    for (int j = 0; j < 4; ++j) st4(hrow + static_cast<long>(k0 + j) * dv + c0, ld4(sD + (k0 + j) * LDV + c0));
    float p[4][4];
    rows_times_state(sK, sD, half, ty, c0, p);
    if (half == 1) {
#pragma unroll
      for (int a = 0; a < 4; ++a) st4(sX + (ty + 16 * a) * LDV + c0, make_float4(p[a][0], p[a][1], p[a][2], p[a][3]));
    }
    __syncthreads();   // k~ has been read by everybody
    if (i > 0) stage_ck(sK, kt + (chunk - 1) * C * DK);
    cp_async_commit();
    if (half == 0) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int r = ty + 16 * a;
        const float4 x = ld4(sX + r * LDV + c0);
        const float4 tv = make_float4(e[a].x + (p[a][0] + x.x), e[a].y + (p[a][1] + x.y), e[a].z + (p[a][2] + x.z), e[a].w + (p[a][3] + x.w));
        st4(du + (tok + r) * dv + col + c0, tv);
        st4(sT + r * LDV + c0, tv);
      }
    }
    cp_async_wait<1>();
    __syncthreads();
    // dS before the chunk = gamma dS + q~^T d_o - w^T (total d v_new); nothing flows into the previous document
    float acc[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 d = ld4(sD + (k0 + j) * LDV + c0);
      acc[j][0] = g * d.x; acc[j][1] = g * d.y; acc[j][2] = g * d.z; acc[j][3] = g * d.w;
    }
    transposed_times_rows(sQ, sO, k0, c0, 1.f, acc);
    transposed_times_rows(sW, sT, k0, c0, -1.f, acc);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      st4(sD + (k0 + j) * LDV + c0, cut ? make_float4(0.f, 0.f, 0.f, 0.f)
                                        : make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]));
  }
  cp_async_wait<0>();
}

// ------------------------------------------------------------------------------------------- from the histories
constexpr int kColTile = 128;   // dv columns per step / CTA
constexpr int kStateSmem = (C * LDK + DK * LDK) * 4;

// rows of a [*, dv] block, columns [c, c + 128), zero past dv
__device__ __forceinline__ void load_cols(float* dst, const float* __restrict__ src, int rows, int dv, int c) {
  for (int i = threadIdx.x; i < rows * (kColTile / 4); i += THREADS) {
    const int r = i >> 5, cc = (i & 31) * 4;
    st4(dst + r * LDK + cc, c + cc < dv ? ld4(src + static_cast<long>(r) * dv + c + cc) : make_float4(0.f, 0.f, 0.f, 0.f));
  }
}

// o = q~ S of one chunk and head, 128 columns per CTA: four rows x (4 + 4) columns a thread
__global__ void __launch_bounds__(THREADS, 2)
gdn_state_out_kernel(const float* __restrict__ qt, const float* __restrict__ hist, float* __restrict__ o, int n, int dv) {
  extern __shared__ __align__(16) float smem[];
  float* sQ = smem;
  float* sS = sQ + C * LDK;
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, c = blockIdx.z * kColTile;
  const long chunk = static_cast<long>(blockIdx.y) * n + blockIdx.x;
  for (int i = tid; i < C * DK / 4; i += THREADS) st4(sQ + (i >> 5) * LDK + (i & 31) * 4, ld4(qt + chunk * C * DK + i * 4));
  load_cols(sS, hist + chunk * DK * dv, DK, dv, c);
  __syncthreads();
  float4 acc[4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a) acc[a][0] = acc[a][1] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (int kk = 0; kk < DK; kk += 4) {
    float4 x[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) x[a] = ld4(sQ + (4 * ty + a) * LDK + kk);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 s0 = ld4(sS + (kk + j) * LDK + 4 * tx), s1 = ld4(sS + (kk + j) * LDK + 64 + 4 * tx);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float s = j == 0 ? x[a].x : j == 1 ? x[a].y : j == 2 ? x[a].z : x[a].w;
        acc[a][0].x += s * s0.x; acc[a][0].y += s * s0.y; acc[a][0].z += s * s0.z; acc[a][0].w += s * s0.w;
        acc[a][1].x += s * s1.x; acc[a][1].y += s * s1.y; acc[a][1].z += s * s1.z; acc[a][1].w += s * s1.w;
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int cc = c + 64 * b + 4 * tx;
      if (cc < dv) st4(o + (chunk * C + 4 * ty + a) * dv + cc, acc[a][b]);
    }
}

// acc[a][b] += A[ty + 16 a] . B[tx + 16 b] over the columns of a tile (A [C][LDK], B [DK][LDK])
__device__ __forceinline__ void rows_dot_rows(float (&acc)[4][8], const float* A, const float* B, int ty, int tx, int cols) {
#pragma unroll 2
  for (int c = 0; c < cols; c += 4) {
    float4 x[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) x[a] = ld4(A + (ty + 16 * a) * LDK + c);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const float4 y = ld4(B + (tx + 16 * b) * LDK + c);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        acc[a][b] = fmaf(x[a].x, y.x, acc[a][b]);
        acc[a][b] = fmaf(x[a].y, y.y, acc[a][b]);
        acc[a][b] = fmaf(x[a].z, y.z, acc[a][b]);
        acc[a][b] = fmaf(x[a].w, y.w, acc[a][b]);
      }
    }
  }
}
__device__ __forceinline__ void store_ck(float* __restrict__ dst, const float (&acc)[4][8], float sign, int ty, int tx) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) dst[(ty + 16 * a) * DK + tx + 16 * b] = sign * acc[a][b];
}

// Gradients of one chunk and head: dw = -du S^T, dq~ = d_o S^T, dk~ = v_new dS^T, dgamma = <dS, S>
__global__ void __launch_bounds__(THREADS, 2)
gdn_state_grad_kernel(const float* __restrict__ vnew, const float* __restrict__ hist, const float* __restrict__ dhist,
                      const float* __restrict__ du, const float* __restrict__ d_o, float* __restrict__ dw,
                      float* __restrict__ dq, float* __restrict__ dk, float* __restrict__ dgamma, int n, int dv) {
  extern __shared__ __align__(16) float smem[];
  float* sA = smem;
  float* sS = sA + C * LDK;
  __shared__ float red[THREADS / 32];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const long chunk = static_cast<long>(blockIdx.y) * n + blockIdx.x;
  const long rows = chunk * C * dv, state = chunk * DK * dv, out = chunk * C * DK;
  float dot = 0.f;
  // three passes over dv; a head of at most 128 columns keeps S for the second
  float acc[4][8] = {};
  for (int c = 0; c < dv; c += kColTile) {
    if (c > 0) __syncthreads();
    load_cols(sS, hist + state, DK, dv, c);
    load_cols(sA, du + rows, C, dv, c);
    __syncthreads();
    rows_dot_rows(acc, sA, sS, ty, tx, min(kColTile, dv - c));
  }
  store_ck(dw + out, acc, -1.f, ty, tx);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[a][b] = 0.f;
  for (int c = 0; c < dv; c += kColTile) {
    __syncthreads();
    if (dv > kColTile) load_cols(sS, hist + state, DK, dv, c);
    load_cols(sA, d_o + rows, C, dv, c);
    __syncthreads();
    rows_dot_rows(acc, sA, sS, ty, tx, min(kColTile, dv - c));
  }
  store_ck(dq + out, acc, 1.f, ty, tx);
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int b = 0; b < 8; ++b) acc[a][b] = 0.f;
  for (int c = 0; c < dv; c += kColTile) {
    __syncthreads();
    for (int i = tid; i < DK * (kColTile / 4); i += THREADS) {
      const int r = i >> 5, cc = (i & 31) * 4;
      float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c + cc < dv) {
        d = ld4(dhist + state + static_cast<long>(r) * dv + c + cc);
        const float4 s = dv > kColTile ? ld4(hist + state + static_cast<long>(r) * dv + c + cc) : ld4(sS + r * LDK + cc);
        dot += d.x * s.x + d.y * s.y + d.z * s.z + d.w * s.w;
      }
      st4(sS + r * LDK + cc, d);   // its own element: read just before by the same thread
    }
    load_cols(sA, vnew + rows, C, dv, c);
    __syncthreads();
    rows_dot_rows(acc, sA, sS, ty, tx, min(kColTile, dv - c));
  }
  store_ck(dk + out, acc, 1.f, ty, tx);
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, m);
  if ((tid & 31) == 0) red[tid >> 5] = dot;
  __syncthreads();
  if (tid == 0) {
    float s = 0.f;
#pragma unroll
    for (int m = 0; m < THREADS / 32; ++m) s += red[m];
    dgamma[chunk] = s;
  }
}

template <typename K>
static int allow(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess ? 0 : -3;
}

}  // namespace b200

#define F(x) static_cast<const float*>(x)
#define FM(x) static_cast<float*>(x)

// All tensors fp32 and contiguous: w, qt, kt [H, n, 64, 128]; u, vnew, o, d_* [H, n, 64, dv]; gamma [H, n];
// reset [n] int32; hist [H, n, 128, dv].  dv must be a multiple of 32.  Returns 0, or a negative code.
extern "C" int b200_gdn_scan_fwd(const void* w, const void* u, const void* qt, const void* kt, const void* gamma,
                                 const void* reset, void* vnew, void* o, void* hist, int H, int n, int dk, int dv,
                                 cudaStream_t st) {
  using namespace b200;
  if (dk != DK || dv % DVT != 0 || dv <= 0 || H > 65535 || dv > 65535) return -2;
  if (H <= 0 || n <= 0) return 0;
  static const int ok = allow(gdn_scan_fwd_kernel, kScanFwdSmem) | allow(gdn_state_out_kernel, kStateSmem);
  if (ok != 0) return ok;
  gdn_scan_fwd_kernel<<<dim3(H, dv / DVT), THREADS, kScanFwdSmem, st>>>(F(w), F(u), F(kt), F(gamma), static_cast<const int*>(reset),
                                                                        FM(vnew), FM(hist), n, dv);
  gdn_state_out_kernel<<<dim3(n, H, (dv + kColTile - 1) / kColTile), THREADS, kStateSmem, st>>>(F(qt), F(hist), FM(o), n, dv);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// du [H, n, 64, dv]; dw, dq, dk [H, n, 64, 128]; dgamma [H, n]; dhist [H, n, 128, dv] work space.
extern "C" int b200_gdn_scan_bwd(const void* w, const void* qt, const void* kt, const void* gamma, const void* reset,
                                 const void* vnew, const void* hist, const void* d_vnew, const void* d_o, void* du,
                                 void* dw, void* dq, void* dk_out, void* dgamma, void* dhist, int H, int n, int dk, int dv,
                                 cudaStream_t st) {
  using namespace b200;
  if (dk != DK || dv % DVT != 0 || dv <= 0 || H > 65535) return -2;
  if (H <= 0 || n <= 0) return 0;
  static const int ok = allow(gdn_scan_bwd_kernel, kScanBwdSmem) | allow(gdn_state_grad_kernel, kStateSmem);
  if (ok != 0) return ok;
  gdn_scan_bwd_kernel<<<dim3(H, dv / DVT), THREADS, kScanBwdSmem, st>>>(F(w), F(qt), F(kt), F(gamma), static_cast<const int*>(reset),
                                                                        F(d_vnew), F(d_o), FM(du), FM(dhist), n, dv);
  gdn_state_grad_kernel<<<dim3(n, H), THREADS, kStateSmem, st>>>(F(vnew), F(hist), F(dhist), F(du), F(d_o), FM(dw), FM(dq), FM(dk_out),
                                                                 FM(dgamma), n, dv);
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}
