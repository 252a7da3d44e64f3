// Streaming and row kernels of the training step: everything the reference
// generates as GLSL in kernels.make_kernels (kernels.py:699-862) and
// tkernels.make_transformer_kernels (tkernels.py:17-389).  All are HBM-bound;
// accesses are coalesced and vectorised where alignment allows, reductions are
// warp/CTA shuffles, and the column sums are deterministic (fixed-order partial
// sums in caller-provided scratch) instead of float atomics.
#include "common.cuh"

#include <algorithm>

namespace {

constexpr int TPB = 256;

// ---- flat elementwise -------------------------------------------------------

__global__ void k_bias_act(const float* __restrict__ acc, const float* __restrict__ bias,
                           float* __restrict__ z, __half* __restrict__ y16, int64_t n, int ncol,
                           int act) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    float v = acc[i] + bias[i % ncol];
    if (z) z[i] = v;
    if (y16) y16[i] = __float2half_rn(vkg_act(v, act));
  }
}

__global__ void k_bias_act_bwd(const float* __restrict__ dy, const float* __restrict__ z,
                               __half* __restrict__ dz16, float* __restrict__ dz32, int64_t n,
                               int act) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    float g = dy[i] * vkg_dact(z[i], act);
    if (dz16) dz16[i] = __float2half_rn(g);
    if (dz32) dz32[i] = g;
  }
}

__global__ void k_cast16(const float* __restrict__ src, __half* __restrict__ dst, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) dst[i] = __float2half_rn(src[i]);
}

__global__ void k_cast16_v4(const float4* __restrict__ src, uint2* __restrict__ dst, int64_t n4) {
  pdl_trigger();
  pdl_wait();
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n4; i += stride) {
    float4 v = src[i];
    __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    uint2 o;
    o.x = *reinterpret_cast<uint32_t*>(&a);
    o.y = *reinterpret_cast<uint32_t*>(&b);
    dst[i] = o;
  }
}

__global__ void k_residual(const float* __restrict__ acc, const float* __restrict__ bias,
                           const float* __restrict__ res, float* __restrict__ out, int64_t n, int D) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) out[i] = res[i] + acc[i] + bias[i % D];
}

__global__ void k_add(const float* __restrict__ a, const float* __restrict__ b,
                      float* __restrict__ out, __half* __restrict__ out16, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    float v = a[i] + b[i];
    if (out) out[i] = v;
    if (out16) out16[i] = __float2half_rn(v);
  }
}

__global__ void k_add_bias(float* __restrict__ x, const float* __restrict__ bias, int64_t n,
                           int ncol) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) x[i] += bias[i % ncol];
}

__global__ void k_grad_add(const float* __restrict__ g, float* __restrict__ arena, int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) arena[i] += g[i];
}

__global__ void k_grad_pull(const float* __restrict__ arena, float* __restrict__ g, int64_t n,
                            float scale) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) g[i] = arena[i] * scale;
}

template <typename T16>
__global__ void k_pack16(const float* __restrict__ src, T16* __restrict__ dst, int64_t n,
                         float scale) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) dst[i] = T16(src[i] * scale);
}

template <typename T16>
__global__ void k_unpack16(const T16* __restrict__ src, float* __restrict__ dst, int64_t n,
                           float scale) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) dst[i] = float(src[i]) * scale;
}

// ---- the same, four values per thread and access -------------------------------------------
//
// 16-byte aligned fp32 matrices whose width is a multiple of four: everything a thread reads is
// requested before anything is used, and the column of a value comes from the launch shape instead
// of a 64-bit remainder.  Bound by issue and latency at these sizes (L2-resident).  1024 x 3072: bias + GELU
// 10.5 -> 5.2 us, GELU' 7.7 -> 4.7; 1024 x 768: residual 5.4 -> 2.6, add 4.9 -> 2.8.

__device__ __forceinline__ uint2 pack4_h(const float4& v) {
  const __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}

constexpr int V4_ROWS = 4;       // rows per thread
// rows x ncol4 float4, blocks of 64 column groups x 4 * V4_ROWS rows: out-of-place op(row element,
// bias element, second operand)
enum { V4_BIAS_ACT, V4_RESIDUAL, V4_ADD_BIAS };
template <int OP>
__global__ void __launch_bounds__(TPB)
k_rows_v4(const float4* a, const float4* __restrict__ bias, const float4* res,
          float4* out, uint2* __restrict__ out16, int nrow, int ncol4, int act) {
  pdl_trigger();
  pdl_wait();
  const int c = blockIdx.x * 64 + (threadIdx.x & 63);
  if (c >= ncol4) return;
  const float4 b = bias[c];
  for (int r0 = (blockIdx.y * 4 + (threadIdx.x >> 6)) * V4_ROWS; r0 < nrow; r0 += gridDim.y * 4 * V4_ROWS) {
    float4 v[V4_ROWS], w[V4_ROWS];
#pragma unroll
    for (int u = 0; u < V4_ROWS; ++u)
      if (r0 + u < nrow) {
        v[u] = a[(int64_t)(r0 + u) * ncol4 + c];
        if (OP == V4_RESIDUAL) w[u] = res[(int64_t)(r0 + u) * ncol4 + c];
      }
#pragma unroll
    for (int u = 0; u < V4_ROWS; ++u) {
      if (r0 + u >= nrow) break;
      const int64_t i = (int64_t)(r0 + u) * ncol4 + c;
      if (OP == V4_RESIDUAL) {
        out[i] = add4(add4(w[u], v[u]), b);
        continue;
      }
      float4 z = add4(v[u], b);
      if (out) out[i] = z;
      if (OP == V4_BIAS_ACT && out16) {
        if (act == VKG_ACT_GELU)
          z = make_float4(vkg_gelu(z.x), vkg_gelu(z.y), vkg_gelu(z.z), vkg_gelu(z.w));
        else
          z = make_float4(vkg_act(z.x, act), vkg_act(z.y, act), vkg_act(z.z, act), vkg_act(z.w, act));
        out16[i] = pack4_h(z);
      }
    }
  }
}

// flat: dz = dy * act'(z) (ACT_BWD) or out = a + b, fp32 and / or fp16 out
enum { V4_ACT_BWD, V4_ADD };
template <int OP>
__global__ void __launch_bounds__(TPB)
k_flat_v4(const float4* a, const float4* b, float4* out,
          uint2* __restrict__ out16, int64_t n4, int act) {
  constexpr int U = 2;
  pdl_trigger();
  pdl_wait();
  const int64_t step = (int64_t)gridDim.x * TPB;
  for (int64_t i0 = (int64_t)blockIdx.x * TPB + threadIdx.x; i0 < n4; i0 += U * step) {
    float4 x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * step < n4) {
        x[u] = a[i0 + u * step];
        y[u] = b[i0 + u * step];
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = i0 + u * step;
      if (i >= n4) break;
      float4 v;
      if (OP == V4_ADD) {
        v = add4(x[u], y[u]);
      } else if (act == VKG_ACT_GELU) {
        v = make_float4(x[u].x * vkg_dgelu(y[u].x), x[u].y * vkg_dgelu(y[u].y), x[u].z * vkg_dgelu(y[u].z),
                        x[u].w * vkg_dgelu(y[u].w));
      } else {
        v = make_float4(x[u].x * vkg_dact(y[u].x, act), x[u].y * vkg_dact(y[u].y, act),
                        x[u].z * vkg_dact(y[u].z, act), x[u].w * vkg_dact(y[u].w, act));
      }
      if (out) out[i] = v;
      if (out16) out16[i] = pack4_h(v);
    }
  }
}

// Head permutes, four values of a head per thread.  A block covers 64 groups of the D / 4 in a
// (rows, D) matrix x 4 * PERM_ROWS rows; which = blockIdx.z picks q, k or v where there are three.
// 1024 x 768: split_qkv 7.9 -> 3.1 us, merge_qkv 7.5 -> 3.4, merge and split 7.3 -> 2.3.
constexpr int PERM_ROWS = 4;
enum { PERM_SPLIT_QKV, PERM_MERGE_QKV, PERM_MERGE, PERM_SPLIT };
template <int OP>
__global__ void __launch_bounds__(TPB)
k_heads_v4(const float* __restrict__ s0, const float* __restrict__ s1, const float* __restrict__ s2,
           __half* __restrict__ d0, __half* __restrict__ d1, __half* __restrict__ d2, int rows, int D, int T,
           int H, int hd) {
  pdl_trigger();
  pdl_wait();
  const int d = (blockIdx.x * 64 + (threadIdx.x & 63)) * 4;
  if (d >= D) return;
  const int which = blockIdx.z;
  const int h = d / hd, j = d - h * hd;
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (OP == PERM_SPLIT_QKV) b = *reinterpret_cast<const float4*>(s1 + which * D + d);     // s1: bias
  const float* src = OP == PERM_MERGE_QKV ? (which == 0 ? s0 : which == 1 ? s1 : s2) : s0;
  __half* dst = OP == PERM_SPLIT_QKV ? (which == 0 ? d0 : which == 1 ? d1 : d2) : d0;
  const int r0 = (blockIdx.y * 4 + (threadIdx.x >> 6)) * PERM_ROWS;
  float4 v[PERM_ROWS];
  int64_t by_head[PERM_ROWS];
#pragma unroll
  for (int u = 0; u < PERM_ROWS; ++u) {
    const int r = r0 + u;
    if (r >= rows) break;
    const int bb = r / T, t = r - bb * T;
    by_head[u] = ((int64_t)(bb * H + h) * T + t) * hd + j;
    const int64_t from = OP == PERM_SPLIT_QKV ? (int64_t)r * 3 * D + which * D + d
                         : OP == PERM_SPLIT   ? (int64_t)r * D + d
                                              : by_head[u];
    v[u] = *reinterpret_cast<const float4*>(src + from);
  }
#pragma unroll
  for (int u = 0; u < PERM_ROWS; ++u) {
    const int r = r0 + u;
    if (r >= rows) break;
    const int64_t to = OP == PERM_MERGE_QKV ? (int64_t)r * 3 * D + which * D + d
                       : OP == PERM_MERGE   ? (int64_t)r * D + d
                                            : by_head[u];
    *reinterpret_cast<uint2*>(dst + to) = pack4_h(OP == PERM_SPLIT_QKV ? add4(v[u], b) : v[u]);
  }
}

// ---- head permutes ------------------------------------------------------------

__global__ void k_split_qkv(const float* __restrict__ qkv, const float* __restrict__ bias,
                            __half* __restrict__ q16, __half* __restrict__ k16,
                            __half* __restrict__ v16, int64_t n, int D, int T, int H, int hd) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int d = (int)(i % D);
    int64_t bt = i / D;
    int t = (int)(bt % T);
    int64_t b = bt / T;
    int h = d / hd, j = d % hd;
    int64_t dst = ((b * H + h) * T + t) * hd + j;
    int64_t src = bt * 3 * D + d;
    q16[dst] = __float2half_rn(qkv[src] + bias[d]);
    k16[dst] = __float2half_rn(qkv[src + D] + bias[d + D]);
    v16[dst] = __float2half_rn(qkv[src + 2 * D] + bias[d + 2 * D]);
  }
}

__global__ void k_merge_qkv_grad(const float* __restrict__ dq, const float* __restrict__ dk,
                                 const float* __restrict__ dv, __half* __restrict__ dqkv16,
                                 int64_t n, int D, int T, int H, int hd) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int d = (int)(i % D);
    int64_t bt = i / D;
    int t = (int)(bt % T);
    int64_t b = bt / T;
    int h = d / hd, j = d % hd;
    int64_t src = ((b * H + h) * T + t) * hd + j;
    int64_t dst = bt * 3 * D + d;
    dqkv16[dst] = __float2half_rn(dq[src]);
    dqkv16[dst + D] = __float2half_rn(dk[src]);
    dqkv16[dst + 2 * D] = __float2half_rn(dv[src]);
  }
}

__global__ void k_merge_heads(const float* __restrict__ src, __half* __restrict__ y16, int64_t n,
                              int D, int T, int H, int hd) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int d = (int)(i % D);
    int64_t bt = i / D;
    int t = (int)(bt % T);
    int64_t b = bt / T;
    int h = d / hd, j = d % hd;
    y16[i] = __float2half_rn(src[((b * H + h) * T + t) * hd + j]);
  }
}

__global__ void k_split_heads(const float* __restrict__ src, __half* __restrict__ dst16, int64_t n,
                              int D, int T, int H, int hd) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int d = (int)(i % D);
    int64_t bt = i / D;
    int t = (int)(bt % T);
    int64_t b = bt / T;
    int h = d / hd, j = d % hd;
    dst16[((b * H + h) * T + t) * hd + j] = __float2half_rn(src[i]);
  }
}

// ---- embeddings -----------------------------------------------------------------

__global__ void k_embed(const float* __restrict__ tok, const float* __restrict__ pos,
                        const uint32_t* __restrict__ ids, const uint32_t* __restrict__ seg,
                        float* __restrict__ x, int64_t n, int D, int T) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int d = (int)(i % D);
    int64_t bt = i / D;
    int t = (int)(bt % T);
    if (seg) t -= (int)seg[bt];
    x[i] = tok[(int64_t)ids[bt] * D + d] + pos[(int64_t)t * D + d];
  }
}

__global__ void k_embed_bwd(const float* __restrict__ dx, const uint32_t* __restrict__ ids,
                            const uint32_t* __restrict__ seg, float* __restrict__ dtok,
                            float* __restrict__ dpos, int64_t n, int D, int T) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    int d = (int)(i % D);
    int64_t bt = i / D;
    int t = (int)(bt % T);
    if (seg) t -= (int)seg[bt];
    float g = dx[i];
    atomicAdd(dtok + (int64_t)ids[bt] * D + d, g);
    atomicAdd(dpos + (int64_t)t * D + d, g);
  }
}

// Four columns per thread (D a multiple of 4, 16-byte aligned tables): one 16-byte access
// per operand, and one 16-byte vector atomic per table in the backward.
__global__ void k_embed_v4(const float4* __restrict__ tok, const float4* __restrict__ pos,
                           const uint32_t* __restrict__ ids, const uint32_t* __restrict__ seg,
                           float4* __restrict__ x, int n4, int D4, int T) {
  pdl_trigger();
  pdl_wait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) {
    const int bt = i / D4, d = i - bt * D4;
    int t = bt % T;
    if (seg) t -= (int)seg[bt];
    const float4 a = tok[(int64_t)ids[bt] * D4 + d], b = pos[(int64_t)t * D4 + d];
    x[i] = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
  }
}

__global__ void k_gather_rows(const float4* __restrict__ src, const uint32_t* __restrict__ rows,
                              float4* __restrict__ dst, int D4) {
  pdl_trigger();
  pdl_wait();
  const float4* from = src + (int64_t)rows[blockIdx.x] * D4;
  for (int d = threadIdx.x; d < D4; d += blockDim.x) dst[(int64_t)blockIdx.x * D4 + d] = from[d];
}

__global__ void k_embed_bwd_v4(const float4* __restrict__ dx, const uint32_t* __restrict__ ids,
                               const uint32_t* __restrict__ seg, float4* __restrict__ dtok,
                               float4* __restrict__ dpos, int n4, int D4, int T) {
  pdl_trigger();
  pdl_wait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) {
    const int bt = i / D4, d = i - bt * D4;
    int t = bt % T;
    if (seg) t -= (int)seg[bt];
    const float4 g = dx[i];
    atomicAdd(dtok + (int64_t)ids[bt] * D4 + d, g);
    atomicAdd(dpos + (int64_t)t * D4 + d, g);
  }
}

// Deterministic scatter-add of the embedding backward (the reference adds with float atomics,
// tkernels.py:317-360, whose order changes from run to run).  Rows that hit the same table
// row are linked into a chain in row order; the warp that owns a chain's first row walks it,
// adds the rows in that order in registers and updates the table row once.
//
// Table `which`: 0 the token table (key = ids[r]), 1 the position table (key = r % T, minus
// the start of the row's packed sample).  keys[which][rows_p] (rows_p = rows rounded up to 4,
// the padding holds -2), next[which][rows] = the next row with r's key or -1,
// has_prev[which][rows] = 1 when an earlier row has it.
__device__ __forceinline__ int embed_key(int which, int r, const uint32_t* ids, const uint32_t* seg,
                                         int T) {
  if (which == 0) return (int)ids[r];
  int t = r % T;
  if (seg) t -= (int)seg[r];
  return t;
}

__global__ void k_embed_keys(const uint32_t* __restrict__ ids, const uint32_t* __restrict__ seg,
                             int* __restrict__ keys, int* __restrict__ has_prev, int rows, int rows_p,
                             int T) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * rows_p) return;
  const int which = i / rows_p, r = i - which * rows_p;
  keys[i] = r < rows ? embed_key(which, r, ids, seg, T) : -2;
  if (r < rows) has_prev[which * rows + r] = 0;
}

// One warp per (table, row): the lanes look through the later rows 128 keys at a time (one
// 16-byte load each) and stop at the first chunk that holds the row's key; the smallest such
// row is the successor, whatever the timing.
__global__ void __launch_bounds__(256)
k_embed_chain(const int* __restrict__ keys, int* __restrict__ next, int* __restrict__ has_prev,
              int rows, int rows_p) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= 2 * rows) return;
  const int which = w / rows, r = w - which * rows;
  const int* k = keys + (size_t)which * rows_p;
  const int key = k[r];
  int found = -1;
  // four chunks of 128 keys per round: the four loads are independent, so a round costs one
  // memory round trip instead of four
  for (int j0 = ((r + 1) & ~3) + lane * 4; found < 0; j0 += 512) {
    unsigned m[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u * 128;
      m[u] = 0;
      if (j < rows_p) {
        const int4 v = *reinterpret_cast<const int4*>(k + j);
        m[u] = (v.x == key && j > r ? 1u : 0u) | (v.y == key && j + 1 > r ? 2u : 0u) |
               (v.z == key && j + 2 > r ? 4u : 0u) | (v.w == key && j + 3 > r ? 8u : 0u);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const unsigned any = __ballot_sync(0xffffffffu, m[u] != 0u);
      if (any && found < 0) {
        const int src = __ffs(any) - 1;
        const int mine = j0 + u * 128 + __ffs(m[u]) - 1;     // meaningful on lane `src` only
        found = __shfl_sync(0xffffffffu, mine, src);
      }
    }
    if (__all_sync(0xffffffffu, j0 + 512 - lane * 4 >= rows_p)) break;   // the warp is past the end
  }
  if (lane == 0) {
    next[which * rows + r] = found;
    if (found >= 0) has_prev[which * rows + found] = 1;   // one writer: its predecessor
  }
}

// A lane has four columns of every 128; of the last 128 those that are left of D.
template <int NV>
__global__ void __launch_bounds__(256)
k_embed_bwd_chain(const float* __restrict__ dx, const uint32_t* __restrict__ ids,
                  const uint32_t* __restrict__ seg, const int* __restrict__ next,
                  const int* __restrict__ has_prev, float* __restrict__ dtok, float* __restrict__ dpos,
                  int rows, int D, int T) {
  pdl_trigger();
  pdl_wait();
  const int which = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r0 = blockIdx.x * (blockDim.x >> 5) + warp;
  if (r0 >= rows || has_prev[which * rows + r0]) return;
  const bool last = ((NV - 1) * 32 + lane) * 4 < D;
  float4 acc[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  // The links of a chain (8 bytes per row, in L1) are followed a few rows ahead of the rows
  // themselves, which are then requested together: with one row per round a chain of 21 (2048
  // bytes over 96 symbols) cost 21 trips to L2; 21.8 -> 10.5 us.
  constexpr int U = NV <= 4 ? 4 : 2;
  for (int r = r0; r >= 0;) {
    int at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      at[u] = r;
      if (r >= 0) r = next[which * rows + r];
    }
    float4 g[U][NV];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0)
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (i < NV - 1 || last)
            g[u][i] = *reinterpret_cast<const float4*>(dx + (size_t)at[u] * D + (i * 32 + lane) * 4);
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (at[u] >= 0)
#pragma unroll
        for (int i = 0; i < NV; ++i)
          if (i < NV - 1 || last) acc[i] = add4(acc[i], g[u][i]);
  }
  float* row = (which == 0 ? dtok : dpos) + (size_t)embed_key(which, r0, ids, seg, T) * D;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    if (i == NV - 1 && !last) break;
    float4* p = reinterpret_cast<float4*>(row + (i * 32 + lane) * 4);
    float4 v = *p;
    v.x += acc[i].x; v.y += acc[i].y; v.z += acc[i].z; v.w += acc[i].w;
    *p = v;
  }
}

// ---- column sums ------------------------------------------------------------------

// The reference's col_sum: one thread per column over fp32 rows (kernels.py:753).
__global__ void k_col_sum(const float* __restrict__ g, float* __restrict__ sums, int ncol,
                          int nrow) {
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncol) return;
  float s = 0.f;
  for (int r = 0; r < nrow; ++r) s += g[(int64_t)r * ncol + c];
  sums[c] = s;
}

constexpr int CS_WARPS = 8;

template <typename T> struct ColVec;
template <> struct ColVec<__half> {   // 8 columns per lane: one 16-byte load per row
  static constexpr int N = 8;
  __device__ static void add(const __half* p, float* s) {
    uint4 u = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&u);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float2 f = __half22float2(h[j]);
      s[2 * j] += f.x;
      s[2 * j + 1] += f.y;
    }
  }
};
template <> struct ColVec<float> {    // 4 columns per lane
  static constexpr int N = 4;
  __device__ static void add(const float* p, float* s) {
    float4 u = *reinterpret_cast<const float4*>(p);
    s[0] += u.x; s[1] += u.y; s[2] += u.z; s[3] += u.w;
  }
};

// Stage 1: block (cx, chunk) sums rows [chunk*rpc, ...) of its 32*N columns into
// partial[chunk][col].  Warps stride the rows; each lane owns N adjacent columns and
// reads them with one 16-byte load per row (scalar loads when ncol is not a multiple
// of N or the base is unaligned).
template <typename T>
__device__ __forceinline__ void col_sum_block(const T* __restrict__ g, float* __restrict__ partial, int ncol,
                                              int nrow, int rows_per_chunk, int vec_ok, int cx, int chunk,
                                              float (*red)[32 * ColVec<T>::N + 1]) {
  constexpr int N = ColVec<T>::N;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = (cx * 32 + lane) * N;
  const int r0 = chunk * rows_per_chunk;
  const int r1 = min(nrow, r0 + rows_per_chunk);
  float s[N];
#pragma unroll
  for (int j = 0; j < N; ++j) s[j] = 0.f;
  if (vec_ok) {
    if (c < ncol) {
      int r = r0 + warp;
      for (; r + 3 * CS_WARPS < r1; r += 4 * CS_WARPS) {   // four rows in flight per lane
        ColVec<T>::add(g + (int64_t)r * ncol + c, s);
        ColVec<T>::add(g + (int64_t)(r + CS_WARPS) * ncol + c, s);
        ColVec<T>::add(g + (int64_t)(r + 2 * CS_WARPS) * ncol + c, s);
        ColVec<T>::add(g + (int64_t)(r + 3 * CS_WARPS) * ncol + c, s);
      }
      for (; r < r1; r += CS_WARPS) ColVec<T>::add(g + (int64_t)r * ncol + c, s);
    }
  } else {
    for (int r = r0 + warp; r < r1; r += CS_WARPS)
#pragma unroll
      for (int j = 0; j < N; ++j)
        if (c + j < ncol) s[j] += float(g[(int64_t)r * ncol + c + j]);
  }
#pragma unroll
  for (int j = 0; j < N; ++j) red[warp][lane * N + j] = s[j];
  __syncthreads();
  for (int t = threadIdx.x; t < 32 * N; t += CS_WARPS * 32) {
    float a = 0.f;
#pragma unroll
    for (int w = 0; w < CS_WARPS; ++w) a += red[w][t];
    int col = cx * 32 * N + t;
    if (col < ncol) partial[(int64_t)chunk * ncol + col] = a;
  }
}

template <typename T>
__global__ void __launch_bounds__(CS_WARPS * 32)
k_col_sum_partial(const T* __restrict__ g, float* __restrict__ partial, int ncol, int nrow, int rows_per_chunk,
                  int vec_ok) {
  __shared__ float red[CS_WARPS][32 * ColVec<T>::N + 1];
  pdl_trigger();
  pdl_wait();
  col_sum_block<T>(g, partial, ncol, nrow, rows_per_chunk, vec_ok, blockIdx.x, blockIdx.y, red);
}

// Stage 2: fixed-order sum of the partials.  A CTA owns 32 columns; its 8 warps each
// add every 8th chunk, then the eight slices are added in order.
constexpr int CSF_SLICES = 8;
__device__ __forceinline__ void col_sum_final_block(const float* __restrict__ partial, float* __restrict__ sums,
                                                    int ncol, int nchunk, int accumulate, int cx,
                                                    float (*red)[32]) {
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int c = cx * 32 + lane;
  float s = 0.f;
  if (c < ncol)
    for (int k = slice; k < nchunk; k += CSF_SLICES) s += partial[(int64_t)k * ncol + c];
  red[slice][lane] = s;
  __syncthreads();
  if (slice == 0 && c < ncol) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < CSF_SLICES; ++k) t += red[k][lane];
    sums[c] = accumulate ? sums[c] + t : t;
  }
}

__global__ void __launch_bounds__(32 * CSF_SLICES)
k_col_sum_final(const float* __restrict__ partial, float* __restrict__ sums, int ncol, int nchunk,
                int accumulate) {
  __shared__ float red[CSF_SLICES][32];
  pdl_trigger();
  pdl_wait();
  col_sum_final_block(partial, sums, ncol, nchunk, accumulate, blockIdx.x, red);
}

// Both stages for several matrices at once (the bias gradients of a small model's layers): a block
// finds its matrix by its number.  Two launches instead of two per layer, the same sums.
constexpr int CSM_MAX = 32;      // matrices per launch: 32 * 56 bytes of arguments
struct ColSumJob {
  const void* g;
  float *partial, *sums;
  int ncol, nrow, rows_per_chunk, nchunk;
  int f16, vec_ok, first1, first2;      // first block of each stage
};
struct ColSumJobs {
  int n, accumulate;
  ColSumJob e[CSM_MAX];
};

__global__ void __launch_bounds__(CS_WARPS * 32)
k_col_sum_partial_multi(const __grid_constant__ ColSumJobs jobs) {
  __shared__ float red[CS_WARPS][32 * ColVec<__half>::N + 1];
  pdl_trigger();
  pdl_wait();
  int e = 0;
  while (e + 1 < jobs.n && (int)blockIdx.x >= jobs.e[e + 1].first1) ++e;
  const ColSumJob& j = jobs.e[e];
  const int b = (int)blockIdx.x - j.first1, chunk = b % j.nchunk, cx = b / j.nchunk;
  if (j.f16)
    col_sum_block<__half>((const __half*)j.g, j.partial, j.ncol, j.nrow, j.rows_per_chunk, j.vec_ok, cx, chunk, red);
  else
    col_sum_block<float>((const float*)j.g, j.partial, j.ncol, j.nrow, j.rows_per_chunk, j.vec_ok, cx, chunk,
                         reinterpret_cast<float(*)[32 * ColVec<float>::N + 1]>(red));
}

__global__ void __launch_bounds__(32 * CSF_SLICES)
k_col_sum_final_multi(const __grid_constant__ ColSumJobs jobs) {
  __shared__ float red[CSF_SLICES][32];
  pdl_trigger();
  pdl_wait();
  int e = 0;
  while (e + 1 < jobs.n && (int)blockIdx.x >= jobs.e[e + 1].first2) ++e;
  const ColSumJob& j = jobs.e[e];
  col_sum_final_block(j.partial, j.sums, j.ncol, j.nchunk, jobs.accumulate, (int)blockIdx.x - j.first2, red);
}

// ---- softmax + cross entropy ---------------------------------------------------------

// Running maximum m and sum s of exp(x - m): one more value, or another such pair.  Written out to the
// last rounding: the two kernels below have to give the same bits, and which of two products goes
// into an fma is otherwise the compiler's choice in each of them.
__device__ __forceinline__ void ce_take(float v, float& m, float& s) {
  if (v > m) {
    s = __fmaf_rn(s, __expf(m - v), 1.0f);
    m = v;
  } else {
    s = __fadd_rn(s, __expf(v - m));
  }
}
__device__ __forceinline__ void ce_merge(float& m, float& s, float m2, float s2) {
  const float mm = fmaxf(m, m2);
  s = __fmaf_rn(s, __expf(m - mm), __fmul_rn(s2, __expf(m2 - mm)));
  m = mm;
}

// One CTA per row.  Online max/sum in one pass, then one pass writing the
// gradient; the second read of the row comes out of L2.
__global__ void __launch_bounds__(TPB)
k_softmax_ce(const float* __restrict__ logits, const uint32_t* __restrict__ labels,
             const float* __restrict__ w, __half* __restrict__ dl16, float* __restrict__ dl32,
             float* __restrict__ loss, int stride, int ncls, float grad_scale) {
  __shared__ float s_m[TPB / 32], s_s[TPB / 32];
  __shared__ float s_logz;
  const int row = blockIdx.x;
  const float* x = logits + (int64_t)row * stride;
  __half* d16 = dl16 ? dl16 + (int64_t)row * stride : nullptr;
  float* d32 = dl32 ? dl32 + (int64_t)row * stride : nullptr;
  float wi = grad_scale;
  if (w) {
    // per-row weights replace the mean; a non-zero grad_scale then is a static loss scale
    wi = w[row] * (grad_scale != 0.0f ? grad_scale : 1.0f);
    if (wi == 0.0f) {
      for (int c = threadIdx.x; c < stride; c += TPB) {
        if (d16) d16[c] = __float2half_rn(0.f);
        if (d32) d32[c] = 0.f;
      }
      if (threadIdx.x == 0) loss[row] = 0.f;
      return;
    }
  }
  float m = -1e30f, s = 0.f;
  for (int c = threadIdx.x; c < ncls; c += TPB) ce_take(x[c], m, s);
  // combine (m, s) pairs across the warp, then across warps
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
    ce_merge(m, s, m2, s2);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    s_m[warp] = m;
    s_s[warp] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float mm = s_m[0], ss = s_s[0];
    for (int k = 1; k < TPB / 32; ++k) ce_merge(mm, ss, s_m[k], s_s[k]);
    float logz = mm + logf(ss);
    s_logz = logz;
    loss[row] = logz - x[labels[row]];
  }
  __syncthreads();
  const float logz = s_logz;
  const int y = (int)labels[row];
  for (int c = threadIdx.x; c < stride; c += TPB) {
    float gv = 0.f;
    if (c < ncls) gv = (__expf(x[c] - logz) - (c == y ? 1.0f : 0.0f)) * wi;
    if (d16) d16[c] = __float2half_rn(gv);
    if (d32) d32[c] = gv;
  }
}

// Narrow rows (a byte-level vocabulary, a classifier's head): one warp per row, the row in
// registers, NV values per lane; a block per row spent its time on two barriers and eight idle
// warps (2048 rows: 96 logits 11.6 -> 4.9 us, 256 logits 12.1 -> 7.1).  It adds in k_softmax_ce's
// order -- columns c and c + 256 in one chain, 32 columns by a butterfly, the eight groups of 32 in
// turn -- so that the results are the same bits: fp16 gradients without a loss scale are small
// enough for the last bit of a row's normaliser to show in the weights.
template <int NV>
__global__ void __launch_bounds__(128)
k_softmax_ce_warp(const float* __restrict__ logits, const uint32_t* __restrict__ labels,
                  const float* __restrict__ w, __half* __restrict__ dl16, float* __restrict__ dl32,
                  float* __restrict__ loss, int rows, int stride, int ncls, float grad_scale) {
  constexpr int NG = NV < 8 ? NV : 8;
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31, row = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= rows) return;
  const int y = (int)labels[row];
  const float* x = logits + (size_t)row * stride;
  float wi = grad_scale;
  bool skip = false;
  if (w) {
    wi = w[row] * (grad_scale != 0.0f ? grad_scale : 1.0f);
    skip = wi == 0.0f;
  }
  float v[NV], m[NG], s[NG];
#pragma unroll
  for (int i = 0; i < NV; ++i) v[i] = i * 32 + lane < ncls ? x[i * 32 + lane] : 0.f;
#pragma unroll
  for (int i = 0; i < NG; ++i) {
    m[i] = -1e30f;
    s[i] = 0.f;
  }
#pragma unroll
  for (int i = 0; i < NV; ++i)
    if (i * 32 + lane < ncls) ce_take(v[i], m[i % NG], s[i % NG]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int i = 0; i < NG; ++i) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m[i], o);
      const float s2 = __shfl_xor_sync(0xffffffffu, s[i], o);
      ce_merge(m[i], s[i], m2, s2);
    }
#pragma unroll
  for (int i = 1; i < NG; ++i) ce_merge(m[0], s[0], m[i], s[i]);
  const float logz = __shfl_sync(0xffffffffu, m[0] + logf(s[0]), 0);
  if (lane == 0) loss[row] = skip ? 0.f : logz - x[y];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = i * 32 + lane;
    if (c >= stride) continue;
    const float g = skip || c >= ncls ? 0.f : (__expf(v[i] - logz) - (c == y ? 1.0f : 0.0f)) * wi;
    if (dl16) dl16[(size_t)row * stride + c] = __float2half_rn(g);
    if (dl32) dl32[(size_t)row * stride + c] = g;
  }
}

// Register-resident variant for wide rows (the GPT head: 50 272 columns): one CTA of
// 768 threads per row, every thread keeps up to NV float4 of the row in registers, so
// the logits are read from HBM exactly once and the gradient is written from registers.
constexpr int CE_THREADS = 768;

template <int NV>
__global__ void __launch_bounds__(CE_THREADS)
k_softmax_ce_reg(const float* __restrict__ logits, const uint32_t* __restrict__ labels,
                 const float* __restrict__ w, __half* __restrict__ dl16, float* __restrict__ dl32,
                 float* __restrict__ loss, int stride, int ncls, float grad_scale, int pf_rows) {
  pdl_trigger();
  pdl_wait();
  __shared__ float s_red[CE_THREADS / 32];
  __shared__ float s_bcast;
  const int row = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const float* x = logits + (size_t)row * stride;
  const int n4 = stride >> 2;
  float wi = grad_scale;
  bool skip = false;
  if (w) {
    wi = w[row] * (grad_scale != 0.0f ? grad_scale : 1.0f);
    skip = wi == 0.0f;
  }
  float4 v[NV];
  float m = -1e30f;
  if (!skip) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c4 = tid + i * CE_THREADS;
      v[i] = c4 < n4 ? *reinterpret_cast<const float4*>(x + 4 * c4) : make_float4(0, 0, 0, 0);
      const int c = 4 * c4;
      if (c + 0 < ncls) m = fmaxf(m, v[i].x);
      if (c + 1 < ncls) m = fmaxf(m, v[i].y);
      if (c + 2 < ncls) m = fmaxf(m, v[i].z);
      if (c + 3 < ncls) m = fmaxf(m, v[i].w);
    }
  }
  // Only one CTA of this size fits an SM, so its load, reduce and store phases do not
  // overlap: pull the row that the CTA after this one on the same SM will want into L2
  // now, which keeps HBM streaming while this row is reduced and written.
  if (row + pf_rows < (int)gridDim.x) {
    const char* nx = reinterpret_cast<const char*>(logits + (size_t)(row + pf_rows) * stride);
    for (int o = tid * 128; o < stride * 4; o += CE_THREADS * 128)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + o));
  }
  m = warp_max(m);
  if (lane == 0) s_red[warp] = m;
  __syncthreads();
  if (warp == 0) {
    float t = lane < CE_THREADS / 32 ? s_red[lane] : -1e30f;
    t = warp_max(t);
    if (lane == 0) s_bcast = t;
  }
  __syncthreads();
  m = s_bcast;
  float sum = 0.f;
  if (!skip) {
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = 4 * (tid + i * CE_THREADS);
      // keep exp(x - m) in place of x: it is what the gradient needs
      v[i].x = c + 0 < ncls ? __expf(v[i].x - m) : 0.f;
      v[i].y = c + 1 < ncls ? __expf(v[i].y - m) : 0.f;
      v[i].z = c + 2 < ncls ? __expf(v[i].z - m) : 0.f;
      v[i].w = c + 3 < ncls ? __expf(v[i].w - m) : 0.f;
      sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    }
  }
  sum = warp_sum(sum);
  __syncthreads();
  if (lane == 0) s_red[warp] = sum;
  __syncthreads();
  if (warp == 0) {
    float t = warp_sum(lane < CE_THREADS / 32 ? s_red[lane] : 0.f);
    if (lane == 0) s_bcast = t;
  }
  __syncthreads();
  sum = s_bcast;
  const int y = (int)labels[row];
  if (tid == 0) loss[row] = skip ? 0.f : (m + logf(sum)) - x[y];
  const float k = skip ? 0.f : wi / sum;
  __half* d16 = dl16 ? dl16 + (size_t)row * stride : nullptr;
  float* d32 = dl32 ? dl32 + (size_t)row * stride : nullptr;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c4 = tid + i * CE_THREADS;
    if (c4 >= n4) continue;
    const int c = 4 * c4;
    float4 g = skip ? make_float4(0, 0, 0, 0)
                    : make_float4(v[i].x * k, v[i].y * k, v[i].z * k, v[i].w * k);
    if (!skip && y >= c && y < c + 4) {
      if (y == c) g.x -= wi;
      else if (y == c + 1) g.y -= wi;
      else if (y == c + 2) g.z -= wi;
      else g.w -= wi;
    }
    if (d16) {
      __half2 a = __floats2half2_rn(g.x, g.y), b = __floats2half2_rn(g.z, g.w);
      uint2 u;
      u.x = *reinterpret_cast<uint32_t*>(&a);
      u.y = *reinterpret_cast<uint32_t*>(&b);
      *reinterpret_cast<uint2*>(d16 + c) = u;
    }
    if (d32) *reinterpret_cast<float4*>(d32 + c) = g;
  }
}

// ---- layernorm ----------------------------------------------------------------------------

// One warp per row, lanes stride the row (the reference's layout, tkernels.py:32-54).
__global__ void k_layernorm(const float* __restrict__ x, const float* __restrict__ gamma,
                            const float* __restrict__ beta, __half* __restrict__ y16,
                            float* __restrict__ mu, float* __restrict__ rstd, int rows, int D) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;
  const float* xr = x + (int64_t)row * D;
  float s = 0.f;
  for (int d = lane; d < D; d += 32) s += xr[d];
  const float m = warp_sum(s) / (float)D;
  float v = 0.f;
  for (int d = lane; d < D; d += 32) {
    float t = xr[d] - m;
    v += t * t;
  }
  const float r = rsqrtf(warp_sum(v) / (float)D + 1e-5f);
  if (lane == 0) {
    mu[row] = m;
    rstd[row] = r;
  }
  __half* yr = y16 + (int64_t)row * D;
  for (int d = lane; d < D; d += 32) yr[d] = __float2half_rn((xr[d] - m) * r * gamma[d] + beta[d]);
}

// D = 128 * NV: the row lives in registers (NV float4 per lane), one read of x.
template <int NV>
__global__ void k_layernorm_vec(const float* __restrict__ x, const float* __restrict__ gamma,
                                const float* __restrict__ beta, __half* __restrict__ y16,
                                float* __restrict__ mu, float* __restrict__ rstd, int rows) {
  constexpr int D = NV * 128;
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;
  const float* xr = x + (size_t)row * D;
  float4 v[NV];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i] = *reinterpret_cast<const float4*>(xr + (i * 32 + lane) * 4);
    s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
  }
  const float m = warp_sum(s) * (1.0f / D);
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    v[i].x -= m; v[i].y -= m; v[i].z -= m; v[i].w -= m;
    q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
  }
  const float r = rsqrtf(warp_sum(q) * (1.0f / D) + 1e-5f);
  if (lane == 0) {
    mu[row] = m;
    rstd[row] = r;
  }
  __half* yr = y16 + (size_t)row * D;
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = (i * 32 + lane) * 4;
    const float4 g = *reinterpret_cast<const float4*>(gamma + c);
    const float4 b = *reinterpret_cast<const float4*>(beta + c);
    __half2 lo = __floats2half2_rn(v[i].x * r * g.x + b.x, v[i].y * r * g.y + b.y);
    __half2 hi = __floats2half2_rn(v[i].z * r * g.z + b.z, v[i].w * r * g.w + b.w);
    uint2 u;
    u.x = *reinterpret_cast<uint32_t*>(&lo);
    u.y = *reinterpret_cast<uint32_t*>(&hi);
    *reinterpret_cast<uint2*>(yr + c) = u;
  }
}

constexpr int LNB_WARPS = 4;

// One column's share of a row's two sums, and the row's gradient there.  Written out to the last
// rounding, because two kernels share it and have to give the same bits: left to the compiler, which
// of two products goes into an fma may differ from one to the next.
__device__ __forceinline__ void ln_bwd_take(float dxh, float xh, float& s1, float& s2) {
  s1 = __fadd_rn(s1, dxh);
  s2 = __fmaf_rn(dxh, xh, s2);
}
__device__ __forceinline__ float ln_bwd_dx(float dy, float gamma, float xh, float r, float s1, float s2, float inv) {
  const float centred = __fmaf_rn(dy, gamma, -__fmul_rn(s1, inv));
  return __fmul_rn(r, __fmaf_rn(-__fmul_rn(xh, s2), inv, centred));
}

// Backward.  Each CTA owns a contiguous band of rows; warp w handles rows
// band0+w, band0+w+4, ...  Per-column partial sums of dy*xhat and dy are kept
// in the warp's private shared-memory strip, combined across the CTA's warps
// and written to scratch[block][2][D]; k_ln_param_final adds the blocks up in
// a fixed order.
__global__ void __launch_bounds__(LNB_WARPS * 32)
k_layernorm_bwd(const float* __restrict__ dy, const float* __restrict__ x,
                const float* __restrict__ gamma, const float* __restrict__ mu,
                const float* __restrict__ rstd, const float* __restrict__ dres,
                float* __restrict__ dx, __half* __restrict__ dx16, __half* __restrict__ dyxh16,
                __half* __restrict__ dy16, float* __restrict__ scratch, int rows, int D,
                int rows_per_block) {
  extern __shared__ float acc[];  // [LNB_WARPS][2][D] when scratch != nullptr
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* a_g = acc + (size_t)warp * 2 * D;
  float* a_b = a_g + D;
  if (scratch) {
    for (int d = lane; d < D; d += 32) {
      a_g[d] = 0.f;
      a_b[d] = 0.f;
    }
  }
  const int r0 = blockIdx.x * rows_per_block;
  const int r1 = min(rows, r0 + rows_per_block);
  const float inv = 1.0f / (float)D;
  for (int row = r0 + warp; row < r1; row += LNB_WARPS) {
    const int64_t base = (int64_t)row * D;
    const float m = mu[row], r = rstd[row];
    float s1 = 0.f, s2 = 0.f;
    for (int d = lane; d < D; d += 32) {
      float dyv = dy[base + d];
      float xh = (x[base + d] - m) * r;
      ln_bwd_take(dyv * gamma[d], xh, s1, s2);
      if (dyxh16) dyxh16[base + d] = __float2half_rn(dyv * xh);
      if (dy16) dy16[base + d] = __float2half_rn(dyv);
      if (scratch) {
        a_g[d] += dyv * xh;
        a_b[d] += dyv;
      }
    }
    s1 = warp_sum(s1);
    s2 = warp_sum(s2);
    for (int d = lane; d < D; d += 32) {
      float o = ln_bwd_dx(dy[base + d], gamma[d], (x[base + d] - m) * r, r, s1, s2, inv);
      if (dres) o = __fadd_rn(o, dres[base + d]);
      if (dx) dx[base + d] = o;
      if (dx16) dx16[base + d] = __float2half_rn(o);
    }
  }
  if (scratch) {
    __syncthreads();
    float* out = scratch + (size_t)blockIdx.x * 2 * D;
    for (int d = threadIdx.x; d < 2 * D; d += blockDim.x) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < LNB_WARPS; ++w) s += acc[(size_t)w * 2 * D + d];
      out[d] = s;
    }
  }
}

constexpr int LNF_SLICES = 32;

// Fixed-order reduction of the per-block partials: 32 columns x 32 slices per CTA,
// each slice adds every 32nd block, then the slices are added in order.
__global__ void __launch_bounds__(32 * LNF_SLICES)
k_ln_param_final(const float* __restrict__ scratch, float* __restrict__ dgamma,
                 float* __restrict__ dbeta, float* __restrict__ dxsum, int D, int nblocks,
                 int nparts) {
  __shared__ float red[LNF_SLICES][32];
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane;  // column in [0, nparts*D): gamma, beta, (dx) parts
  const int W = nparts * D;
  float s = 0.f;
  if (c < W)
    for (int k = slice; k < nblocks; k += LNF_SLICES) s += scratch[(size_t)k * W + c];
  red[slice][lane] = s;
  __syncthreads();
  if (slice == 0 && c < W) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < LNF_SLICES; ++k) t += red[k][lane];
    if (c < D) dgamma[c] = t;
    else if (c < 2 * D) dbeta[c - D] = t;
    else dxsum[c - 2 * D] = t;
  }
}

// Vectorised backward for D = 128 * NV: a warp owns a row, each lane holds NV float4
// of x and dy in registers, and keeps its columns' dgamma/dbeta partial sums in
// registers across all the rows it visits.
constexpr int LNV_WARPS = 8;

template <int NV>
__global__ void __launch_bounds__(LNV_WARPS * 32)
k_layernorm_bwd_vec(const float* __restrict__ dy, const float* __restrict__ x,
                    const float* __restrict__ gamma, const float* __restrict__ mu,
                    const float* __restrict__ rstd, const float* __restrict__ dres,
                    float* __restrict__ dx, __half* __restrict__ dx16,
                    float* __restrict__ scratch, int rows, int nparts) {
  constexpr int D = NV * 128;
  pdl_trigger();
  pdl_wait();
  __shared__ float red[LNV_WARPS][32 * 4 + 4];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float4 g[NV], ag[NV], ab[NV], ax[NV];   // ax: column sums of the output (nparts == 3)
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    g[i] = *reinterpret_cast<const float4*>(gamma + (i * 32 + lane) * 4);
    ag[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    ab[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    ax[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float inv = 1.0f / (float)D;
  const int warps_total = gridDim.x * LNV_WARPS;
  for (int row = blockIdx.x * LNV_WARPS + warp; row < rows; row += warps_total) {
    const size_t base = (size_t)row * D;
    const float m = mu[row], r = rstd[row];
    // all three streams of the row are requested before anything is consumed: the kernel
    // holds one CTA per SM (its registers), so memory latency is hidden by loads in flight
    // per warp, not by other warps
    float4 xv[NV], dv[NV], rv[NV];
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      xv[i] = *reinterpret_cast<const float4*>(x + base + (i * 32 + lane) * 4);
      dv[i] = *reinterpret_cast<const float4*>(dy + base + (i * 32 + lane) * 4);
    }
    if (dres) {
#pragma unroll
      for (int i = 0; i < NV; ++i)
        rv[i] = *reinterpret_cast<const float4*>(dres + base + (i * 32 + lane) * 4);
    } else {
#pragma unroll
      for (int i = 0; i < NV; ++i) rv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      xv[i].x = (xv[i].x - m) * r; xv[i].y = (xv[i].y - m) * r;
      xv[i].z = (xv[i].z - m) * r; xv[i].w = (xv[i].w - m) * r;
      float a0 = dv[i].x * g[i].x, a1 = dv[i].y * g[i].y, a2 = dv[i].z * g[i].z, a3 = dv[i].w * g[i].w;
      s1 += a0 + a1 + a2 + a3;
      s2 += a0 * xv[i].x + a1 * xv[i].y + a2 * xv[i].z + a3 * xv[i].w;
      ag[i].x += dv[i].x * xv[i].x; ag[i].y += dv[i].y * xv[i].y;
      ag[i].z += dv[i].z * xv[i].z; ag[i].w += dv[i].w * xv[i].w;
      ab[i].x += dv[i].x; ab[i].y += dv[i].y; ab[i].z += dv[i].z; ab[i].w += dv[i].w;
    }
    s1 = warp_sum(s1) * inv;
    s2 = warp_sum(s2) * inv;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      float4 o;
      o.x = r * (dv[i].x * g[i].x - s1 - xv[i].x * s2);
      o.y = r * (dv[i].y * g[i].y - s1 - xv[i].y * s2);
      o.z = r * (dv[i].z * g[i].z - s1 - xv[i].z * s2);
      o.w = r * (dv[i].w * g[i].w - s1 - xv[i].w * s2);
      const size_t off = base + (i * 32 + lane) * 4;
      o.x += rv[i].x; o.y += rv[i].y; o.z += rv[i].z; o.w += rv[i].w;
      if (dx) *reinterpret_cast<float4*>(dx + off) = o;
      if (dx16) {
        __half2 a = __floats2half2_rn(o.x, o.y), b = __floats2half2_rn(o.z, o.w);
        uint2 u;
        u.x = *reinterpret_cast<uint32_t*>(&a);
        u.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(dx16 + off) = u;
      }
      ax[i].x += o.x; ax[i].y += o.y; ax[i].z += o.z; ax[i].w += o.w;
    }
  }
  if (scratch) {
    // add the CTA's warps in a fixed order, one 128-column group at a time
    float* out = scratch + (size_t)blockIdx.x * nparts * D;
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      if (part >= nparts) break;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        float4 v = part == 0 ? ag[i] : part == 1 ? ab[i] : ax[i];
        __syncthreads();
        *reinterpret_cast<float4*>(&red[warp][lane * 4]) = v;
        __syncthreads();
        if (warp == 0) {
          float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int w = 0; w < LNV_WARPS; ++w) {
            float4 u = *reinterpret_cast<const float4*>(&red[w][lane * 4]);
            t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
          }
          *reinterpret_cast<float4*>(out + part * D + (i * 32 + lane) * 4) = t;
        }
      }
    }
  }
}

// Backward that leaves the parameter sums to column sums over its dy * xhat and dy copies: one warp
// per row, the row in registers.  k_layernorm_bwd reads each row twice, the second time behind the
// reductions: 6.7 -> 4.0 us at 1024 x 768, back to back.  A lane has the columns it has there,
// 32 apart, and adds them in the same order, so the bits are the same.
template <int NV>
__global__ void __launch_bounds__(128)
k_layernorm_bwd_rows(const float* __restrict__ dy, const float* __restrict__ x, const float* __restrict__ gamma,
                     const float* __restrict__ mu, const float* __restrict__ rstd, const float* __restrict__ dres,
                     float* __restrict__ dx, __half* __restrict__ dx16, __half* __restrict__ dyxh16,
                     __half* __restrict__ dy16, int rows) {
  constexpr int D = NV * 128, N = NV * 4;
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;
  const size_t base = (size_t)row * D + lane;
  const float m = mu[row], r = rstd[row], inv = 1.0f / (float)D;
  float xh[N], dv[N], s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    xh[i] = x[base + i * 32];
    dv[i] = dy[base + i * 32];
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    xh[i] = (xh[i] - m) * r;
    ln_bwd_take(dv[i] * gamma[i * 32 + lane], xh[i], s1, s2);
    if (dyxh16) dyxh16[base + i * 32] = __float2half_rn(dv[i] * xh[i]);
    if (dy16) dy16[base + i * 32] = __float2half_rn(dv[i]);
  }
  s1 = warp_sum(s1);
  s2 = warp_sum(s2);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float o = ln_bwd_dx(dv[i], gamma[i * 32 + lane], xh[i], r, s1, s2, inv);
    if (dres) o = __fadd_rn(o, dres[base + i * 32]);
    if (dx) dx[base + i * 32] = o;
    if (dx16) dx16[base + i * 32] = __float2half_rn(o);
  }
}

// ---- attention softmax ---------------------------------------------------------------------

// One warp per (batch*head, query) row; causal; optional packed-sample start.
__global__ void k_attn_softmax(const float* __restrict__ s, const uint32_t* __restrict__ seg,
                               __half* __restrict__ p16, int64_t rows, int T, int H, float scale,
                               int fill_block) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;
  const int64_t base = row * T;
  const int q = (int)(row % T);
  int st = 0;
  if (seg) st = (int)seg[(row / T / H) * T + q];
  float mx = -1e30f;
  for (int j = st + lane; j <= q; j += 32) mx = fmaxf(mx, s[base + j] * scale);
  mx = warp_max(mx);
  float sum = 0.f;
  for (int j = st + lane; j <= q; j += 32) sum += __expf(fmaf(s[base + j], scale, -mx));
  sum = warp_sum(sum);
  const float inv = 1.0f / sum;
  // zeros above the diagonal: to the end of the row, or only to the end of the
  // fill_block-wide tile the consumer's causal K range stops at
  const int jend = fill_block > 0 ? min(T, (q / fill_block + 1) * fill_block) : T;
  for (int j = lane; j < jend; j += 32) {
    float v = 0.f;
    if (j >= st && j <= q) v = __expf(fmaf(s[base + j], scale, -mx)) * inv;
    p16[base + j] = __float2half_rn(v);
  }
}

__global__ void k_attn_softmax_bwd(const float* __restrict__ dp, const __half* __restrict__ p16,
                                   __half* __restrict__ ds16, int64_t rows, int T, float scale,
                                   int fill_block) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
  if (row >= rows) return;
  const int64_t base = row * T;
  const int q = (int)(row % T);
  float dot = 0.f;
  for (int j = lane; j <= q; j += 32) dot = fmaf(dp[base + j], __half2float(p16[base + j]), dot);
  dot = warp_sum(dot);
  const int jend = fill_block > 0 ? min(T, (q / fill_block + 1) * fill_block) : T;
  for (int j = lane; j < jend; j += 32) {
    float v = 0.f;
    if (j <= q) v = __half2float(p16[base + j]) * (dp[base + j] - dot) * scale;
    ds16[base + j] = __float2half_rn(v);
  }
}

// The same with the row in registers (T up to 1024, 32 * NV keys): scores and gradients are read
// once and only up to the diagonal.  Lanes own the same keys and add in the same order as above.
// Issue-bound, not memory-bound: 128 keys at a time are skipped past the diagonal by a branch of
// the whole warp, and a block's (batch * head, rows) come from the launch shape, long rows first.
// 32 heads x 512 x 512: 13.9 -> 9.5 us, backward 10.0 -> 7.7.  (Four keys per lane and access
// add in another order, which loss gradients in fp16 subnormals, without a loss scale, show.)
template <int NV>
__global__ void __launch_bounds__(256)
k_attn_softmax_reg(const float* __restrict__ s, const uint32_t* __restrict__ seg, __half* __restrict__ p16, int T,
                   int H, float scale, int fill_block) {
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = (int)(gridDim.y - 1 - blockIdx.y) * 8 + warp;
  if (q >= T) return;
  const int st = seg ? (int)seg[(blockIdx.x / (unsigned)H) * T + q] : 0;
  const int64_t row = ((int64_t)blockIdx.x * T + q) * T;
  const int keys = q - st, last = keys - lane;      // key 32 * i of this lane counts while 32 * i <= last
  const float* sr = s + row + st + lane;
  __half* pr = p16 + row;
  float v[NV];
#pragma unroll
  for (int g = 0; g < NV; g += 4)
    if (32 * g <= keys)
#pragma unroll
      for (int i = g; i < g + 4; ++i) v[i] = 32 * i <= last ? sr[32 * i] : 0.f;
  float mx = -1e30f, sum = 0.f;
#pragma unroll
  for (int g = 0; g < NV; g += 4)
    if (32 * g <= keys)
#pragma unroll
      for (int i = g; i < g + 4; ++i)
        if (32 * i <= last) mx = fmaxf(mx, v[i] * scale);
  mx = warp_max(mx);
#pragma unroll
  for (int g = 0; g < NV; g += 4)
    if (32 * g <= keys)
#pragma unroll
      for (int i = g; i < g + 4; ++i) {
        v[i] = 32 * i <= last ? __expf(fmaf(v[i], scale, -mx)) : 0.f;
        sum += v[i];
      }
  const float inv = 1.0f / warp_sum(sum);
  const int jend = fill_block > 0 ? min(T, (q / fill_block + 1) * fill_block) : T;
  for (int j = lane; j < min(st, jend); j += 32) pr[j] = __float2half_rn(0.f);
#pragma unroll
  for (int g = 0; g < NV; g += 4) {
    if (st + 32 * g >= jend) break;
#pragma unroll
    for (int i = g; i < g + 4; ++i) {
      const int j = st + lane + 32 * i;
      if (j < jend) pr[j] = __float2half_rn(32 * i <= last ? v[i] * inv : 0.f);
    }
  }
}

template <int NV>
__global__ void __launch_bounds__(256)
k_attn_softmax_bwd_reg(const float* __restrict__ dp, const __half* __restrict__ p16, __half* __restrict__ ds16, int T,
                       float scale, int fill_block) {
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q = (int)(gridDim.y - 1 - blockIdx.y) * 8 + warp;
  if (q >= T) return;
  const int64_t base = ((int64_t)blockIdx.x * T + q) * T + lane;
  const int last = q - lane;
  float d[NV], p[NV];
#pragma unroll
  for (int g = 0; g < NV; g += 4)
    if (32 * g <= q)
#pragma unroll
      for (int i = g; i < g + 4; ++i) {
        d[i] = 32 * i <= last ? dp[base + 32 * i] : 0.f;
        p[i] = 32 * i <= last ? __half2float(p16[base + 32 * i]) : 0.f;
      }
  float dot = 0.f;
#pragma unroll
  for (int g = 0; g < NV; g += 4)
    if (32 * g <= q)
#pragma unroll
      for (int i = g; i < g + 4; ++i) dot = fmaf(d[i], p[i], dot);
  dot = warp_sum(dot);
  const int jend = fill_block > 0 ? min(T, (q / fill_block + 1) * fill_block) : T;
#pragma unroll
  for (int g = 0; g < NV; g += 4) {
    if (32 * g >= jend) break;
#pragma unroll
    for (int i = g; i < g + 4; ++i)
      if (lane + 32 * i < jend)
        ds16[base + 32 * i] = __float2half_rn(32 * i <= last ? p[i] * (d[i] - dot) * scale : 0.f);
  }
}

// ---- AdamW -----------------------------------------------------------------------------------

__device__ __forceinline__ void adamw_one(float& w, float g, float& m, float& v, float lr, float b1,
                                          float b2, float bc1, float bc2, float eps, float wd) {
  m = b1 * m + (1.0f - b1) * g;
  v = b2 * v + (1.0f - b2) * g * g;
  float mh = m / bc1;
  float vh = v / bc2;
  w -= lr * (mh / (sqrtf(vh) + eps) + wd * w);
}

__global__ void k_adamw(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                        float* __restrict__ v, __half* __restrict__ w16,
                        const float* __restrict__ hp, int64_t n, float wd) {
  const float lr = hp[0], b1 = hp[1], b2 = hp[2], bc1 = hp[3], bc2 = hp[4], eps = hp[5];
  const float gs = hp[6] != 0.0f ? hp[6] : 1.0f;
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) {
    float wi = w[i], mi = m[i], vi = v[i];
    adamw_one(wi, g[i] * gs, mi, vi, lr, b1, b2, bc1, bc2, eps, wd);
    w[i] = wi;
    m[i] = mi;
    v[i] = vi;
    if (w16) w16[i] = __float2half_rn(wi);
  }
}

struct AdamTensor {
  float* w;
  const float* g;
  float* m;
  float* v;
  __half* w16;
  int64_t n;
  float wd;
  int pad;
};

// The step-varying scalars of the optimiser (autograd.py:313-323): learning rate, both betas, both
// bias corrections, epsilon, gradient scale, unused.
struct AdamHp {
  float v[8];
};

// One launch for every parameter tensor: block b looks up (tensor, chunk) and updates CHUNK
// elements.  Bound by HBM (30 bytes per parameter) when there are many blocks and by latency when
// there are few, where a thread has one float4 of each array and all of them in flight.
// The scalars arrive as a kernel argument: read by the kernel from the mapped host memory the
// caller keeps them in, they took 15 of the 22 us of a 0.28 M-parameter step (a cold walk over the
// host link).  hp is the fallback for scalars that live in device memory.
template <int CHUNK>
__global__ void __launch_bounds__(TPB)
k_adamw_multi(const AdamTensor* __restrict__ tensors, const int2* __restrict__ blockmap,
              const float* __restrict__ hp, const AdamHp val) {
  pdl_trigger();
  pdl_wait();
  float lr = val.v[0], b1 = val.v[1], b2 = val.v[2], bc1 = val.v[3], bc2 = val.v[4], eps = val.v[5], gs = val.v[6];
  if (hp) {
    lr = hp[0]; b1 = hp[1]; b2 = hp[2]; bc1 = hp[3]; bc2 = hp[4]; eps = hp[5]; gs = hp[6];
  }
  if (gs == 0.0f) gs = 1.0f;
  const int2 bm = blockmap[blockIdx.x];
  const AdamTensor t = tensors[bm.x];
  const int64_t lo = (int64_t)bm.y * CHUNK;
  const int64_t hi = min(t.n, lo + CHUNK);
  const bool vec = (((uintptr_t)t.w | (uintptr_t)t.g | (uintptr_t)t.m | (uintptr_t)t.v) & 15) == 0 &&
                   ((uintptr_t)t.w16 & 7) == 0;
  int64_t tail = lo;                       // elements the vector path leaves over
  if (vec) {
    for (int64_t i = lo + threadIdx.x * 4; i + 3 < hi; i += TPB * 4) {
      float4 w = *reinterpret_cast<float4*>(t.w + i);
      float4 g = *reinterpret_cast<const float4*>(t.g + i);
      float4 m = *reinterpret_cast<float4*>(t.m + i);
      float4 v = *reinterpret_cast<float4*>(t.v + i);
      adamw_one(w.x, g.x * gs, m.x, v.x, lr, b1, b2, bc1, bc2, eps, t.wd);
      adamw_one(w.y, g.y * gs, m.y, v.y, lr, b1, b2, bc1, bc2, eps, t.wd);
      adamw_one(w.z, g.z * gs, m.z, v.z, lr, b1, b2, bc1, bc2, eps, t.wd);
      adamw_one(w.w, g.w * gs, m.w, v.w, lr, b1, b2, bc1, bc2, eps, t.wd);
      *reinterpret_cast<float4*>(t.w + i) = w;
      *reinterpret_cast<float4*>(t.m + i) = m;
      *reinterpret_cast<float4*>(t.v + i) = v;
      if (t.w16) {
        __half2 a = __floats2half2_rn(w.x, w.y), b = __floats2half2_rn(w.z, w.w);
        uint2 o;
        o.x = *reinterpret_cast<uint32_t*>(&a);
        o.y = *reinterpret_cast<uint32_t*>(&b);
        *reinterpret_cast<uint2*>(t.w16 + i) = o;
      }
    }
    tail = lo + ((hi - lo) & ~(int64_t)3);
  }
  for (int64_t i = tail + threadIdx.x; i < hi; i += TPB) {
    float wi = t.w[i], mi = t.m[i], vi = t.v[i];
    adamw_one(wi, t.g[i] * gs, mi, vi, lr, b1, b2, bc1, bc2, eps, t.wd);
    t.w[i] = wi; t.m[i] = mi; t.v[i] = vi;
    if (t.w16) t.w16[i] = __float2half_rn(wi);
  }
}

// Blocks of 4096 elements once those make four resident waves (148 SMs x 8 blocks each), of 1024
// below that, where the number of loads in flight counts.  (All sixteen loads of a 4096 block
// issued at once were 12 % slower at 124 M parameters: registers halve the resident blocks.)
constexpr int ADAM_CHUNK = 4096, ADAM_CHUNK_SMALL = 1024;
constexpr int64_t ADAM_SMALL_MAX = (int64_t)ADAM_CHUNK * 148 * 8 * 4;

struct AdamTable {
  AdamTensor* tensors = nullptr;
  int2* blockmap = nullptr;
  int nblocks = 0;
  int chunk = ADAM_CHUNK;
};

// ---- gradient accumulation over a table of tensors ---------------------------------------------

struct PairTensor {
  float* a;          // the tensor
  float* b;          // its place in the arena
  int64_t n;
};
constexpr int PAIR_CHUNK = 2048;
struct PairTable {
  PairTensor* tensors = nullptr;
  int2* blockmap = nullptr;
  int nblocks = 0;
};

// b += a (PULL false) or a = b * scale (PULL true) for every tensor of the table in one launch: a
// model has a dozen tensors per layer and most of them are a few KB.
template <bool PULL>
__global__ void __launch_bounds__(TPB)
k_pairs_multi(const PairTensor* __restrict__ tensors, const int2* __restrict__ blockmap, float scale) {
  constexpr int U = PAIR_CHUNK / (TPB * 4);
  const int2 bm = blockmap[blockIdx.x];
  const PairTensor t = tensors[bm.x];
  const int64_t lo = (int64_t)bm.y * PAIR_CHUNK, hi = min(t.n, lo + PAIR_CHUNK);
  int64_t tail = lo;
  if ((((uintptr_t)t.a | (uintptr_t)t.b) & 15) == 0) {
    float4 x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = lo + (u * TPB + threadIdx.x) * 4;
      if (i + 3 < hi) {
        y[u] = *reinterpret_cast<const float4*>(t.b + i);
        if (!PULL) x[u] = *reinterpret_cast<const float4*>(t.a + i);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = lo + (u * TPB + threadIdx.x) * 4;
      if (i + 3 >= hi) continue;
      if (PULL)
        *reinterpret_cast<float4*>(t.a + i) =
            make_float4(y[u].x * scale, y[u].y * scale, y[u].z * scale, y[u].w * scale);
      else
        *reinterpret_cast<float4*>(t.b + i) =
            make_float4(y[u].x + x[u].x, y[u].y + x[u].y, y[u].z + x[u].z, y[u].w + x[u].w);
    }
    tail = lo + ((hi - lo) & ~(int64_t)3);
  }
  for (int64_t i = tail + threadIdx.x; i < hi; i += TPB) {
    if (PULL) t.a[i] = t.b[i] * scale;
    else t.b[i] += t.a[i];
  }
}

// Device copies of a table and of its block -> (tensor, chunk) map.
template <typename T, typename Tensor>
int table_upload(T* t, const std::vector<Tensor>& ts, const std::vector<int2>& map) {
  t->nblocks = (int)map.size();
  cudaError_t e = cudaMalloc(&t->tensors, ts.size() * sizeof(Tensor));
  if (e == cudaSuccess) e = cudaMalloc(&t->blockmap, map.size() * sizeof(int2));
  if (e == cudaSuccess)
    e = cudaMemcpy(t->tensors, ts.data(), ts.size() * sizeof(Tensor), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(t->blockmap, map.data(), map.size() * sizeof(int2), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) return 0;
  if (t->tensors) cudaFree(t->tensors);
  if (t->blockmap) cudaFree(t->blockmap);
  VKG_FAIL("tensor table: %s", cudaGetErrorString(e));
}

// Host address of mapped or pinned host memory given by its device address; null for the rest.
const float* host_view(const float* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  return a.type == cudaMemoryTypeHost ? static_cast<const float*>(a.hostPointer) : nullptr;
}

inline unsigned flat_grid(vkg_device* dev, int64_t n) {
  return vkg_blocks(n, TPB, (int64_t)dev->sm_count * 16);
}

}  // namespace

// ---- C ABI -----------------------------------------------------------------------------------

// Launch through vkg_launch, marked short when the work is a few microseconds.
#define VKG_RUN(fam, is_short, kernel, grid, block, ...)                                              \
  VKG_CUDA(vkg_launch(dev, (fam) | vkg_short_if(is_short), kernel, grid, dim3(block), 0, 1, __VA_ARGS__))

static bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr) {
  return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) == 0;
}
constexpr int64_t SHORT_ELEMS = 8 << 20;     // fp32 values a short elementwise launch moves at most
constexpr int64_t SHORT_ROWS = 2 << 20;      // and a short layernorm's rows hold

// Grid of k_rows_v4 over n values in rows of ncol, or false when the vector kernel does not apply.
static bool rows_v4(int64_t n, int ncol, int* nrow, dim3* grid) {
  if (ncol % 4 != 0 || n % ncol != 0 || n / ncol >= (1ll << 30)) return false;
  *nrow = (int)(n / ncol);
  const int per = 4 * V4_ROWS;
  *grid = dim3((unsigned)((ncol / 4 + 63) / 64), (unsigned)std::min((*nrow + per - 1) / per, 65535));
  return true;
}

// Grid of k_heads_v4, or false.
static bool heads_v4(int64_t n, int D, int T, int H, int hd, int which, int* rows, dim3* grid) {
  if (D <= 0 || T <= 0 || hd % 4 != 0 || D != H * hd || n % D != 0) return false;
  const int64_t r = n / D, per = 4 * PERM_ROWS;
  if ((r + per - 1) / per > 65535) return false;
  *rows = (int)r;
  *grid = dim3((unsigned)((D / 4 + 63) / 64), (unsigned)((r + per - 1) / per), (unsigned)which);
  return true;
}

extern "C" int vkg_bias_act(vkg_device* dev, const float* acc, const float* bias, float* z, void* y16,
                            int64_t n, int ncol, int act) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(acc && bias && n > 0 && ncol > 0, "bias_act: bad arguments");
  int nrow;
  dim3 grid;
  if (rows_v4(n, ncol, &nrow, &grid) && aligned16(acc, bias, z) && ((uintptr_t)y16 & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_rows_v4<V4_BIAS_ACT>, grid, TPB, (const float4*)acc, (const float4*)bias,
            nullptr, (float4*)z, (uint2*)y16, nrow, ncol / 4, act);
    return vkg_check_launch("bias_act");
  }
  k_bias_act<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(acc, bias, z, (__half*)y16, n, ncol, act);
  return vkg_check_launch("bias_act");
}

extern "C" int vkg_bias_act_bwd(vkg_device* dev, const float* dy, const float* z, void* dz16,
                                float* dz32, int64_t n, int act) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dy && z && n > 0, "bias_act_bwd: bad arguments");
  if (n % 4 == 0 && aligned16(dy, z, dz32) && ((uintptr_t)dz16 & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_flat_v4<V4_ACT_BWD>, dim3(flat_grid(dev, n / 8)), TPB, (const float4*)dy,
            (const float4*)z, (float4*)dz32, (uint2*)dz16, n / 4, act);
    return vkg_check_launch("bias_act_bwd");
  }
  k_bias_act_bwd<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(dy, z, (__half*)dz16, dz32, n, act);
  return vkg_check_launch("bias_act_bwd");
}

extern "C" int vkg_bias(vkg_device* dev, const float* acc, const float* bias, float* z, int64_t n,
                        int ncol) {
  return vkg_bias_act(dev, acc, bias, z, nullptr, n, ncol, VKG_ACT_NONE);
}

extern "C" int vkg_col_sum(vkg_device* dev, const float* g, float* sums, int ncol, int nrow) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(g && sums && ncol > 0 && nrow > 0, "col_sum: bad arguments");
  k_col_sum<<<vkg_blocks(ncol, 128), 128, 0, dev->stream>>>(g, sums, ncol, nrow);
  return vkg_check_launch("col_sum");
}

static int col_sum_chunks(int ncol, int nrow) {
  int col_blocks = (ncol + 255) / 256;               // the fp16 block width (fp32 blocks are 128)
  int want = (1184 + col_blocks - 1) / col_blocks;   // ~8 CTAs per SM on 148 SMs
  int max_chunks = (nrow + 31) / 32;               // at least 32 rows per chunk
  if (want > max_chunks) want = max_chunks;
  if (want < 1) want = 1;
  if (want > 1024) want = 1024;
  return want;
}

extern "C" int64_t vkg_col_sum_scratch_floats(int ncol, int nrow) {
  if (ncol <= 0 || nrow <= 0) return 0;
  return (int64_t)col_sum_chunks(ncol, nrow) * ncol;
}

int vkg_launch_col_sum_final(vkg_device* dev, const float* partial, float* sums, int ncol, int nchunk,
                             int accumulate) {
  if (dev->defer_finals) {
    dev->finals.push_back(vkg_final_entry{partial, {sums, nullptr, nullptr}, ncol, ncol, nchunk,
                                          accumulate, 0, 0});
    return 0;
  }
  VKG_CUDA(vkg_launch(dev, VKG_K_SMALL | VKG_SHORT, k_col_sum_final, dim3((unsigned)((ncol + 31) / 32)),
                      dim3(32 * CSF_SLICES), 0, 1, partial, sums, ncol, nchunk, accumulate));
  return vkg_check_launch("col_sum_final");
}

extern "C" int vkg_col_sum_det(vkg_device* dev, const void* g, int g_dtype, float* sums,
                               float* scratch, int ncol, int nrow, int accumulate) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(g && sums && scratch && ncol > 0 && nrow > 0, "col_sum_det: bad arguments");
  VKG_REQUIRE(g_dtype == VKG_F32 || g_dtype == VKG_F16, "col_sum_det: dtype must be f32 or f16");
  int nchunk = col_sum_chunks(ncol, nrow);
  int rpc = (nrow + nchunk - 1) / nchunk;
  const int per_block = 32 * (g_dtype == VKG_F16 ? 8 : 4);
  const int vec_ok = (ncol % (per_block / 32) == 0) && (((uintptr_t)g & 15) == 0);
  dim3 grid((ncol + per_block - 1) / per_block, nchunk);
  // The two launches overlap: a single one, whose last block per column group (a counter) adds the
  // partials up, measured 10 us against 4 (1024 x 768) and 17 against 4 (2048 x 768).
  const bool brief = (int64_t)ncol * nrow <= SHORT_ELEMS;
  if (g_dtype == VKG_F16)
    VKG_RUN(VKG_K_SMALL, brief, k_col_sum_partial<__half>, grid, CS_WARPS * 32, (const __half*)g, scratch, ncol, nrow,
            rpc, vec_ok);
  else
    VKG_RUN(VKG_K_SMALL, brief, k_col_sum_partial<float>, grid, CS_WARPS * 32, (const float*)g, scratch, ncol, nrow, rpc,
            vec_ok);
  if (vkg_check_launch("col_sum_partial")) return 1;
  VKG_RUN(VKG_K_SMALL, true, k_col_sum_final, dim3((unsigned)((ncol + 31) / 32)), 32 * CSF_SLICES, scratch, sums, ncol,
          nchunk, accumulate);
  return vkg_check_launch("col_sum_final");
}

extern "C" int vkg_col_sum_multi(vkg_device* dev, int n, const void* const* g, const int32_t* g_dtype,
                                 float* const* sums, const int32_t* ncol, const int32_t* nrow, float* scratch,
                                 int accumulate) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(n > 0 && g && g_dtype && sums && ncol && nrow && scratch, "col_sum_multi: bad arguments");
  for (int at = 0; at < n; at += CSM_MAX) {
    ColSumJobs jobs;
    jobs.n = n - at < CSM_MAX ? n - at : CSM_MAX;
    jobs.accumulate = accumulate;
    int64_t blocks1 = 0, blocks2 = 0, elems = 0;
    for (int i = 0; i < jobs.n; ++i) {
      ColSumJob& j = jobs.e[i];
      j.g = g[at + i];
      j.sums = sums[at + i];
      j.ncol = ncol[at + i];
      j.nrow = nrow[at + i];
      j.f16 = g_dtype[at + i] == VKG_F16;
      VKG_REQUIRE(j.g && j.sums && j.ncol > 0 && j.nrow > 0 && (j.f16 || g_dtype[at + i] == VKG_F32),
                  "col_sum_multi: bad matrix %d", at + i);
      j.partial = scratch;
      j.nchunk = col_sum_chunks(j.ncol, j.nrow);
      j.rows_per_chunk = (j.nrow + j.nchunk - 1) / j.nchunk;
      const int per_lane = j.f16 ? 8 : 4;
      j.vec_ok = j.ncol % per_lane == 0 && ((uintptr_t)j.g & 15) == 0;
      j.first1 = (int)blocks1;
      j.first2 = (int)blocks2;
      blocks1 += (int64_t)((j.ncol + 32 * per_lane - 1) / (32 * per_lane)) * j.nchunk;
      blocks2 += (j.ncol + 31) / 32;
      elems += (int64_t)j.ncol * j.nrow;
      scratch += vkg_col_sum_scratch_floats(j.ncol, j.nrow);
    }
    VKG_REQUIRE(blocks1 < (1ll << 31), "col_sum_multi: too many blocks");
    VKG_RUN(VKG_K_SMALL, elems <= SHORT_ELEMS, k_col_sum_partial_multi, dim3((unsigned)blocks1), CS_WARPS * 32, jobs);
    if (vkg_check_launch("col_sum_partial_multi")) return 1;
    VKG_RUN(VKG_K_SMALL, true, k_col_sum_final_multi, dim3((unsigned)blocks2), 32 * CSF_SLICES, jobs);
    if (vkg_check_launch("col_sum_final_multi")) return 1;
  }
  return 0;
}

// ---- deferred final passes -------------------------------------------------------------
//
// The second stage of a two-stage column sum is a few microseconds of work behind a launch;
// a GPT-2-small backward has 49 of them (layernorm parameters, qkv and fc1 bias gradients),
// each between two large kernels.  While deferral is on they are collected on the host and
// vkg_finals_flush runs them all as ONE launch: the table travels as the kernel's parameter,
// a CTA finds its entry by its block number.  Results do not depend on timing: each column is
// added by 32 slices (slice s takes rows s, s + 32, ...) that are then added in order.
constexpr int FIN_SLICES = 32;
constexpr int FIN_MAX = 64;      // entries per launch: 64 * 56 bytes stay under the 4 KB limit
struct FinalTable {
  int n, reserved;
  vkg_final_entry e[FIN_MAX];
};

__global__ void __launch_bounds__(32 * FIN_SLICES)
k_finals_multi(const __grid_constant__ FinalTable tab) {
  pdl_trigger();
  pdl_wait();
  __shared__ float4 red4[FIN_SLICES][32];
  int e = 0;
  while (e + 1 < tab.n && (int)blockIdx.x >= tab.e[e + 1].first_block) ++e;
  const float* __restrict__ partial = tab.e[e].partial;
  const int W = tab.e[e].W, D = tab.e[e].D, nchunk = tab.e[e].nchunk;
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  if (tab.e[e].reserved) {
    // four columns per lane (W, D multiples of 4, 16-byte aligned rows): a block covers 128
    // columns with one 16-byte load per lane and row.  Per column the order of the additions is
    // the same as below -- slice s takes rows s, s + 32, ..., the slices are added in order.
    const int c = (((int)blockIdx.x - tab.e[e].first_block) * 32 + lane) * 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < W)
      for (int k = slice; k < nchunk; k += FIN_SLICES) {
        const float4 v = *reinterpret_cast<const float4*>(partial + (size_t)k * W + c);
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
    red4[slice][lane] = s;
    __syncthreads();
    if (slice == 0 && c < W) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < FIN_SLICES; ++k) {
        const float4 u = red4[k][lane];
        t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
      }
      float4* d = reinterpret_cast<float4*>(tab.e[e].dst[c / D] + (c % D));
      if (tab.e[e].accumulate) {
        const float4 o = *d;
        t.x += o.x; t.y += o.y; t.z += o.z; t.w += o.w;
      }
      *d = t;
    }
    return;
  }
  float* red = reinterpret_cast<float*>(red4);       // [FIN_SLICES][32] floats
  const int c = ((int)blockIdx.x - tab.e[e].first_block) * 32 + lane;
  float s = 0.f;
  if (c < W)
    for (int k = slice; k < nchunk; k += FIN_SLICES) s += partial[(size_t)k * W + c];
  red[slice * 32 + lane] = s;
  __syncthreads();
  if (slice == 0 && c < W) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < FIN_SLICES; ++k) t += red[k * 32 + lane];
    float* d = tab.e[e].dst[c / D] + (c % D);
    *d = tab.e[e].accumulate ? *d + t : t;
  }
}

extern "C" int vkg_finals_defer(vkg_device* dev, int on) {
  if (vkg_bind(dev)) return 1;
  if (on < 0) dev->finals.clear();     // drop what an abandoned recording left behind
  VKG_REQUIRE(on > 0 || dev->finals.empty(), "finals_defer: %d final passes are pending; call vkg_finals_flush",
              (int)dev->finals.size());
  dev->defer_finals = on > 0;
  return 0;
}

extern "C" int vkg_finals_flush(vkg_device* dev) {
  if (vkg_bind(dev)) return 1;
  dev->defer_finals = false;
  std::vector<vkg_final_entry> todo;
  todo.swap(dev->finals);
  for (size_t i0 = 0; i0 < todo.size(); i0 += FIN_MAX) {
    FinalTable tab;
    memset(&tab, 0, sizeof(tab));
    int blocks = 0;
    for (size_t i = i0; i < todo.size() && i < i0 + FIN_MAX; ++i) {
      vkg_final_entry en = todo[i];
      VKG_REQUIRE(en.partial && en.dst[0] && en.W > 0 && en.D > 0 && en.W <= 3 * en.D && en.nchunk > 0 &&
                      (en.W <= en.D || en.dst[1]) && (en.W <= 2 * en.D || en.dst[2]),
                  "finals_flush: malformed entry");
      en.first_block = blocks;
      // 16-byte columns when every row of the partials and every destination allows it
      bool vec = en.W % 4 == 0 && en.D % 4 == 0 && ((uintptr_t)en.partial & 15) == 0;
      for (int d = 0; d < 3; ++d)
        if (en.dst[d] && ((uintptr_t)en.dst[d] & 15)) vec = false;
      en.reserved = vec ? 1 : 0;
      blocks += vec ? (en.W + 127) / 128 : (en.W + 31) / 32;
      tab.e[tab.n++] = en;
    }
    VKG_RUN(VKG_K_SMALL, true, k_finals_multi, dim3((unsigned)blocks), 32 * FIN_SLICES, tab);
    if (vkg_check_launch("finals_multi")) return 1;
  }
  return 0;
}

// ---- column sums for callers that cannot allocate -----------------------------------
//
// Some hosts of this library may not call cudaMalloc once they are running: a plugin
// loaded into a process whose memory pool is owned by someone else, or a real-time loop
// that must not take the allocator's locks.  For them the partial sums of the
// two-stage column reduction live in a fixed array inside the library image instead
// of caller-provided scratch.  Every GPU that loads the library carries the array
// (4 MiB) until the process exits.
constexpr int64_t COLSUM_STATIC_FLOATS = 1 << 20;
static __device__ __align__(256) float g_colsum_static[COLSUM_STATIC_FLOATS];

namespace {
std::mutex g_colsum_static_mu;
std::map<int, float*> g_colsum_static_ptr;   // device ordinal -> device address of the array

// The array's name is only a host-side handle here; kernels need its device address,
// which differs per device and is looked up once per device with that device current.
int colsum_static_address(vkg_device* dev, float** out) {
  std::lock_guard<std::mutex> lock(g_colsum_static_mu);
  auto it = g_colsum_static_ptr.find(dev->ordinal);
  if (it != g_colsum_static_ptr.end()) {
    *out = it->second;
    return 0;
  }
  if (dev->capturing) {
    // the look-up may load the module, which is not allowed while a stream is being captured
    vkg_set_error("col_sum_static: the first call on a device sets the array's address up and "
                  "must come before any stream capture on that device");
    return 1;
  }
  float* ptr = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void**)&ptr, g_colsum_static);
  if (e != cudaSuccess || ptr == nullptr) {
    vkg_set_error("col_sum_static: cudaGetSymbolAddress failed on device %d: %s", dev->ordinal,
                  cudaGetErrorString(e));
    return 1;
  }
  g_colsum_static_ptr[dev->ordinal] = ptr;
  *out = ptr;
  return 0;
}
}  // namespace

extern "C" int64_t vkg_col_sum_static_max_floats(void) { return COLSUM_STATIC_FLOATS; }

extern "C" int vkg_col_sum_static(vkg_device* dev, const void* g, int g_dtype, float* sums, int ncol,
                                  int nrow, int accumulate) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(g && sums && ncol > 0 && nrow > 0, "col_sum_static: bad arguments");
  VKG_REQUIRE(g_dtype == VKG_F32 || g_dtype == VKG_F16, "col_sum_static: dtype must be f32 or f16");
  const int64_t need = vkg_col_sum_scratch_floats(ncol, nrow);
  VKG_REQUIRE(need <= COLSUM_STATIC_FLOATS,
              "col_sum_static: %d columns x %d rows needs %lld floats of partial sums, the built-in "
              "array holds %lld; use vkg_col_sum_det with your own scratch",
              ncol, nrow, (long long)need, (long long)COLSUM_STATIC_FLOATS);
  float* scratch = nullptr;
  if (colsum_static_address(dev, &scratch)) return 1;
  // Every partial the final pass reads is overwritten by the first pass of this same
  // call, so nothing left behind by an earlier call needs clearing.
  int nchunk = col_sum_chunks(ncol, nrow);
  int rpc = (nrow + nchunk - 1) / nchunk;
  const int per_block = 32 * (g_dtype == VKG_F16 ? 8 : 4);
  const int vec_ok = (ncol % (per_block / 32) == 0) && (((uintptr_t)g & 15) == 0);
  dim3 grid((ncol + per_block - 1) / per_block, nchunk);
  if (g_dtype == VKG_F16)
    k_col_sum_partial<__half><<<grid, CS_WARPS * 32, 0, dev->stream>>>((const __half*)g, scratch,
                                                                        ncol, nrow, rpc, vec_ok);
  else
    k_col_sum_partial<float><<<grid, CS_WARPS * 32, 0, dev->stream>>>((const float*)g, scratch, ncol,
                                                                       nrow, rpc, vec_ok);
  if (vkg_check_launch("col_sum_static partial")) return 1;
  k_col_sum_final<<<(ncol + 31) / 32, 32 * CSF_SLICES, 0, dev->stream>>>(scratch, sums, ncol, nchunk,
                                                                         accumulate);
  return vkg_check_launch("col_sum_static final");
}

extern "C" int vkg_softmax_ce(vkg_device* dev, const float* logits, const uint32_t* labels,
                              const float* w, void* dl16, float* dl32, float* loss, int rows,
                              int stride, int ncls, float grad_scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(logits && labels && loss && rows > 0 && stride >= ncls && ncls > 0,
              "softmax_ce: bad arguments");
  const bool aligned = stride % 4 == 0 && (((uintptr_t)logits | (uintptr_t)dl32) & 15) == 0 &&
                       ((uintptr_t)dl16 & 7) == 0;
  const int n4 = stride / 4;
  if (aligned && n4 > 4 * CE_THREADS && n4 <= 17 * CE_THREADS) {
    // wide rows: one read of the logits, everything else from registers
    const int nv = (n4 + CE_THREADS - 1) / CE_THREADS;
#define VKG_CE(NV)                                                                              \
  VKG_CUDA(vkg_launch(dev, VKG_K_CE, k_softmax_ce_reg<NV>, dim3((unsigned)rows), dim3(CE_THREADS), 0, 1, logits, \
                      labels, w, (__half*)dl16, dl32, loss, stride, ncls, grad_scale,             \
                      dev->sm_count * (NV <= 8 ? 2 : 1)))
    if (nv <= 8) VKG_CE(8);
    else if (nv <= 12) VKG_CE(12);
    else VKG_CE(17);
#undef VKG_CE
    return vkg_check_launch("softmax_ce_reg");
  }
  if (stride <= 1024) {
#define VKG_CE(NV)                                                                                          \
  VKG_RUN(VKG_K_CE, (int64_t)rows * stride <= SHORT_ELEMS, k_softmax_ce_warp<NV>,                           \
          dim3((unsigned)((rows + 3) / 4)), 128, logits, labels, w, (__half*)dl16, dl32, loss, rows,        \
          stride, ncls, grad_scale)
    if (stride <= 32) VKG_CE(1);
    else if (stride <= 64) VKG_CE(2);
    else if (stride <= 128) VKG_CE(4);
    else if (stride <= 256) VKG_CE(8);
    else if (stride <= 512) VKG_CE(16);
    else VKG_CE(32);
#undef VKG_CE
    return vkg_check_launch("softmax_ce_warp");
  }
  k_softmax_ce<<<rows, TPB, 0, dev->stream>>>(logits, labels, w, (__half*)dl16, dl32, loss, stride,
                                              ncls, grad_scale);
  return vkg_check_launch("softmax_ce");
}

extern "C" int vkg_adamw(vkg_device* dev, float* w, const float* g, float* m, float* v, void* w16,
                         const float* hp, int64_t n, float wd) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(w && g && m && v && hp && n > 0, "adamw: bad arguments");
  k_adamw<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(w, g, m, v, (__half*)w16, hp, n, wd);
  return vkg_check_launch("adamw");
}

extern "C" int vkg_adamw_table_create(vkg_device* dev, int ntensors, float* const* w,
                                      const float* const* g, float* const* m, float* const* v,
                                      void* const* w16, const int64_t* n, const float* wd,
                                      void** table) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(ntensors > 0 && w && g && m && v && n && wd && table, "adamw_table: bad arguments");
  std::vector<AdamTensor> ts(ntensors);
  std::vector<int2> map;
  int64_t total = 0;
  for (int i = 0; i < ntensors; ++i) total += n[i];
  const int chunk = total < ADAM_SMALL_MAX ? ADAM_CHUNK_SMALL : ADAM_CHUNK;
  for (int i = 0; i < ntensors; ++i) {
    VKG_REQUIRE(n[i] > 0 && w[i] && g[i] && m[i] && v[i], "adamw_table: tensor %d is empty", i);
    ts[i].w = w[i]; ts[i].g = g[i]; ts[i].m = m[i]; ts[i].v = v[i];
    ts[i].w16 = w16 ? (__half*)w16[i] : nullptr;
    ts[i].n = n[i]; ts[i].wd = wd[i]; ts[i].pad = 0;
    int chunks = (int)((n[i] + chunk - 1) / chunk);
    for (int c = 0; c < chunks; ++c) map.push_back(make_int2(i, c));
  }
  AdamTable* t = new AdamTable();
  t->chunk = chunk;
  if (table_upload(t, ts, map)) {
    delete t;
    return 1;
  }
  *table = t;
  return 0;
}

extern "C" int vkg_adamw_table_destroy(vkg_device* dev, void* table) {
  if (!table) return 0;
  if (vkg_bind(dev)) return 1;
  AdamTable* t = (AdamTable*)table;
  cudaFree(t->tensors);
  cudaFree(t->blockmap);
  delete t;
  return 0;
}

extern "C" int vkg_adamw_multi(vkg_device* dev, void* table, const float* hp) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(table && hp, "adamw_multi: bad arguments");
  AdamTable* t = (AdamTable*)table;
  // A capture that the caller began on this device's stream is not ours to refresh: there the kernel
  // reads the scalars itself, whenever the graph runs.
  cudaStreamCaptureStatus theirs = cudaStreamCaptureStatusNone;
  if (!dev->capturing) VKG_CUDA(cudaStreamIsCapturing(dev->stream, &theirs));
  const float* host = theirs == cudaStreamCaptureStatusNone ? host_view(hp) : nullptr;
  AdamHp val = {};
  if (host) {
    memcpy(val.v, host, 7 * sizeof(float));
    val.v[7] = (float)dev->captured_hp.size();     // which entry of the list this launch belongs to
  }
  VKG_CUDA(vkg_launch(dev, VKG_K_ADAMW | vkg_short_if(t->chunk != ADAM_CHUNK),
                      t->chunk == ADAM_CHUNK ? k_adamw_multi<ADAM_CHUNK> : k_adamw_multi<ADAM_CHUNK_SMALL>,
                      dim3((unsigned)t->nblocks), dim3(TPB), 0, 1, t->tensors, t->blockmap, host ? nullptr : hp, val));
  if (dev->capturing && host) dev->captured_hp.push_back(host);
  return vkg_check_launch("adamw_multi");
}

// A recorded optimiser step takes its scalars afresh whenever the graph is launched: the graph
// keeps the node, its arguments and the host address the scalars are read from.
void vkg_graph_find_hp(vkg_graph* g, const std::vector<const float*>& hps,
                       const std::vector<cudaGraphNode_t>& nodes) {
  for (cudaGraphNode_t node : nodes) {
    cudaGraphNodeType type;
    cudaKernelNodeParams kp;
    if (cudaGraphNodeGetType(node, &type) != cudaSuccess || type != cudaGraphNodeTypeKernel ||
        cudaGraphKernelNodeGetParams(node, &kp) != cudaSuccess)
      continue;
    if (kp.func != (void*)k_adamw_multi<ADAM_CHUNK> && kp.func != (void*)k_adamw_multi<ADAM_CHUNK_SMALL>) continue;
    if (*(const float**)kp.kernelParams[2] != nullptr) continue;      // scalars in device memory
    vkg_graph_hp e;
    e.node = node;
    e.params = kp;
    e.tensors = *(void**)kp.kernelParams[0];
    e.blockmap = *(void**)kp.kernelParams[1];
    const size_t k = (size_t)static_cast<const AdamHp*>(kp.kernelParams[3])->v[7];
    if (k >= hps.size()) continue;
    e.hp = hps[k];
    g->hp.push_back(e);
  }
}

int vkg_graph_refresh_hp(vkg_graph* g) {
  for (vkg_graph_hp& e : g->hp) {
    AdamHp val = {};
    memcpy(val.v, e.hp, 7 * sizeof(float));
    const float* none = nullptr;
    void* args[4] = {&e.tensors, &e.blockmap, &none, &val};
    cudaKernelNodeParams kp = e.params;
    kp.kernelParams = args;
    kp.extra = nullptr;
    VKG_CUDA(cudaGraphExecKernelNodeSetParams(g->exec, e.node, &kp));
  }
  return 0;
}

extern "C" int vkg_grad_table_create(vkg_device* dev, int ntensors, float* const* g, float* const* arena,
                                     const int64_t* n, void** table) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(ntensors > 0 && g && arena && n && table, "grad_table: bad arguments");
  std::vector<PairTensor> ts;
  std::vector<int2> map;
  for (int i = 0; i < ntensors; ++i) {
    VKG_REQUIRE(g[i] && arena[i] && n[i] > 0, "grad_table: tensor %d is empty", i);
    // tensors that follow one another on both sides are one piece
    if (!ts.empty() && ts.back().a + ts.back().n == g[i] && ts.back().b + ts.back().n == arena[i])
      ts.back().n += n[i];
    else
      ts.push_back(PairTensor{g[i], arena[i], n[i]});
  }
  for (size_t i = 0; i < ts.size(); ++i)
    for (int c = 0; c < (int)((ts[i].n + PAIR_CHUNK - 1) / PAIR_CHUNK); ++c) map.push_back(make_int2((int)i, c));
  PairTable* t = new PairTable();
  if (table_upload(t, ts, map)) {
    delete t;
    return 1;
  }
  *table = t;
  return 0;
}

extern "C" int vkg_grad_table_destroy(vkg_device* dev, void* table) {
  if (!table) return 0;
  if (vkg_bind(dev)) return 1;
  PairTable* t = (PairTable*)table;
  cudaFree(t->tensors);
  cudaFree(t->blockmap);
  delete t;
  return 0;
}

extern "C" int vkg_grad_add_multi(vkg_device* dev, void* table) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(table, "grad_add_multi: null table");
  PairTable* t = (PairTable*)table;
  k_pairs_multi<false><<<t->nblocks, TPB, 0, dev->stream>>>(t->tensors, t->blockmap, 1.0f);
  return vkg_check_launch("grad_add_multi");
}

extern "C" int vkg_grad_pull_multi(vkg_device* dev, void* table, float scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(table, "grad_pull_multi: null table");
  PairTable* t = (PairTable*)table;
  k_pairs_multi<true><<<t->nblocks, TPB, 0, dev->stream>>>(t->tensors, t->blockmap, scale);
  return vkg_check_launch("grad_pull_multi");
}

extern "C" int vkg_cast16(vkg_device* dev, const float* src, void* dst16, int64_t n) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(src && dst16 && n > 0, "cast16: bad arguments");
  if ((n & 3) == 0 && (((uintptr_t)src & 15) == 0) && (((uintptr_t)dst16 & 7) == 0)) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_cast16_v4, dim3(flat_grid(dev, n / 4)), TPB, (const float4*)src,
            (uint2*)dst16, n / 4);
  } else {
    k_cast16<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(src, (__half*)dst16, n);
  }
  return vkg_check_launch("cast16");
}

extern "C" int vkg_layernorm(vkg_device* dev, const float* x, const float* gamma, const float* beta,
                             void* y16, float* mu, float* rstd, int rows, int D) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(x && gamma && beta && y16 && mu && rstd && rows > 0 && D > 0, "layernorm: bad arguments");
  const int wpb = 4;
  const bool aligned = ((((uintptr_t)x | (uintptr_t)gamma | (uintptr_t)beta) & 15) == 0) &&
                       (((uintptr_t)y16 & 7) == 0);
  if (aligned && D % 128 == 0 && D <= 1024) {
    const unsigned grid = (rows + wpb - 1) / wpb;
#define VKG_LN(NV)                                                                                                \
  VKG_RUN(VKG_K_LN, (int64_t)rows * D <= SHORT_ROWS, k_layernorm_vec<NV>, dim3(grid), wpb * 32, x, gamma, beta, \
          (__half*)y16, mu, rstd, rows)
    switch (D / 128) {
      case 1: VKG_LN(1); break;
      case 2: VKG_LN(2); break;
      case 3: VKG_LN(3); break;
      case 4: VKG_LN(4); break;
      case 5: VKG_LN(5); break;
      case 6: VKG_LN(6); break;
      case 7: VKG_LN(7); break;
      default: VKG_LN(8); break;
    }
#undef VKG_LN
    return vkg_check_launch("layernorm_vec");
  }
  k_layernorm<<<(rows + wpb - 1) / wpb, wpb * 32, 0, dev->stream>>>(x, gamma, beta, (__half*)y16, mu,
                                                                    rstd, rows, D);
  return vkg_check_launch("layernorm");
}

static int ln_bwd_blocks(int rows) {
  int b = (rows + LNB_WARPS - 1) / LNB_WARPS;  // at least one row per warp
  if (b > 296) b = 296;
  if (b < 1) b = 1;
  return b;
}

extern "C" int64_t vkg_layernorm_bwd_scratch_floats(int rows, int D) {
  if (rows <= 0 || D <= 0) return 0;
  return (int64_t)ln_bwd_blocks(rows) * 3 * D;
}

template <int NV>
static void launch_ln_bwd_vec(vkg_device* dev, int nblocks, const float* dy, const float* x,
                              const float* gamma, const float* mu, const float* rstd,
                              const float* dres, float* dx, void* dx16, float* scratch, int rows,
                              int nparts) {
  // a failed launch is picked up by the caller's vkg_check_launch
  vkg_launch(dev, VKG_K_LN_BWD | vkg_short_if((int64_t)rows * NV * 128 <= SHORT_ROWS), k_layernorm_bwd_vec<NV>,
             dim3((unsigned)nblocks), dim3(LNV_WARPS * 32), 0, 1, dy, x, gamma, mu, rstd, dres, dx, (__half*)dx16,
             scratch, rows, nparts);
}

extern "C" int vkg_layernorm_bwd(vkg_device* dev, const float* dy, const float* x, const float* gamma,
                                 const float* mu, const float* rstd, const float* dres, float* dx,
                                 void* dx16, void* dyxh16, void* dy16, float* dgamma, float* dbeta,
                                 float* dxsum, float* scratch, int rows, int D) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dy && x && gamma && mu && rstd && rows > 0 && D > 0, "layernorm_bwd: bad arguments");
  const bool fused = dgamma != nullptr || dbeta != nullptr;
  if (fused) VKG_REQUIRE(dgamma && dbeta && scratch, "layernorm_bwd: dgamma, dbeta and scratch go together");
  const int nparts = dxsum ? 3 : 2;
  VKG_REQUIRE(!dxsum || (fused && D % 128 == 0 && D <= 1024 && !dyxh16 && !dy16),
              "layernorm_bwd: dxsum needs dgamma/dbeta and D a multiple of 128 up to 1024");
  int nblocks = ln_bwd_blocks(rows);
  const bool aligned = ((((uintptr_t)dy | (uintptr_t)x | (uintptr_t)gamma | (uintptr_t)dres |
                          (uintptr_t)dx | (uintptr_t)scratch) & 15) == 0) && (((uintptr_t)dx16 & 7) == 0);
  if (D % 128 == 0 && D <= 1024 && !fused && aligned && (dyxh16 || dy16)) {
#define VKG_LNR(NV)                                                                                           \
  VKG_RUN(VKG_K_LN_BWD, (int64_t)rows * D <= SHORT_ROWS, k_layernorm_bwd_rows<NV>,                            \
          dim3((unsigned)((rows + 3) / 4)), 128, dy, x, gamma, mu, rstd, dres, dx, (__half*)dx16,             \
          (__half*)dyxh16, (__half*)dy16, rows)
    switch (D / 128) {
      case 1: VKG_LNR(1); break;
      case 2: VKG_LNR(2); break;
      case 3: VKG_LNR(3); break;
      case 4: VKG_LNR(4); break;
      case 5: VKG_LNR(5); break;
      case 6: VKG_LNR(6); break;
      case 7: VKG_LNR(7); break;
      default: VKG_LNR(8); break;
    }
#undef VKG_LNR
    return vkg_check_launch("layernorm_bwd_rows");
  }
  if (D % 128 == 0 && D <= 1024 && !dyxh16 && !dy16 && aligned) {
    // register-resident rows; every CTA writes its partial sums (possibly zero)
    int nb = (rows + LNV_WARPS - 1) / LNV_WARPS;
    if (nb > nblocks) nb = nblocks;
    // from D = 640 on a CTA's registers (three row streams and three sets of column sums per
    // lane) leave room for one CTA per SM only: a second CTA per SM would run as a second wave
    if (D >= 640 && nb > dev->sm_count) nb = dev->sm_count;
    float* sc = fused ? scratch : nullptr;
    switch (D / 128) {
      case 1: launch_ln_bwd_vec<1>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      case 2: launch_ln_bwd_vec<2>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      case 3: launch_ln_bwd_vec<3>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      case 4: launch_ln_bwd_vec<4>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      case 5: launch_ln_bwd_vec<5>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      case 6: launch_ln_bwd_vec<6>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      case 7: launch_ln_bwd_vec<7>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
      default: launch_ln_bwd_vec<8>(dev, nb, dy, x, gamma, mu, rstd, dres, dx, dx16, sc, rows, nparts); break;
    }
    if (vkg_check_launch("layernorm_bwd_vec")) return 1;
    nblocks = nb;
  } else {
    int rpb = (rows + nblocks - 1) / nblocks;
    nblocks = (rows + rpb - 1) / rpb;
    size_t smem = fused ? (size_t)LNB_WARPS * 2 * D * sizeof(float) : 0;
    VKG_REQUIRE(smem <= 48 * 1024, "layernorm_bwd: fused parameter sums support D <= %d",
                48 * 1024 / (LNB_WARPS * 8));
    k_layernorm_bwd<<<nblocks, LNB_WARPS * 32, smem, dev->stream>>>(
        dy, x, gamma, mu, rstd, dres, dx, (__half*)dx16, (__half*)dyxh16, (__half*)dy16,
        fused ? scratch : nullptr, rows, D, rpb);
    if (vkg_check_launch("layernorm_bwd")) return 1;
  }
  if (fused) {
    VKG_REQUIRE(!dxsum || (D % 128 == 0 && D <= 1024 && aligned),
                "layernorm_bwd: dxsum needs 16-byte aligned operands");
    if (dev->defer_finals) {
      dev->finals.push_back(vkg_final_entry{scratch, {dgamma, dbeta, dxsum}, nparts * D, D, nblocks,
                                            0, 0, 0});
      return 0;
    }
    k_ln_param_final<<<(nparts * D + 31) / 32, 32 * LNF_SLICES, 0, dev->stream>>>(
        scratch, dgamma, dbeta, dxsum, D, nblocks, nparts);
    return vkg_check_launch("ln_param_final");
  }
  return 0;
}

extern "C" int vkg_attn_softmax(vkg_device* dev, const float* s, const uint32_t* seg, void* p16,
                                int64_t rows, int T, int H, float scale, int fill_block) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(s && p16 && rows > 0 && T > 0, "attn_softmax: bad arguments");
  const int wpb = 8;
  if (T <= 1024 && rows % T == 0 && rows / T < (1ll << 31)) {
#define VKG_SM(NV)                                                                                          \
  VKG_RUN(VKG_K_SMALL, rows * T <= SHORT_ELEMS, k_attn_softmax_reg<NV>,                                     \
          dim3((unsigned)(rows / T), (unsigned)((T + 7) / 8)), 256, s, seg, (__half*)p16, T, H > 0 ? H : 1, \
          scale, fill_block)
    if (T <= 128) VKG_SM(4);
    else if (T <= 256) VKG_SM(8);
    else if (T <= 512) VKG_SM(16);
    else VKG_SM(32);
#undef VKG_SM
    return vkg_check_launch("attn_softmax");
  }
  k_attn_softmax<<<(unsigned)((rows + wpb - 1) / wpb), wpb * 32, 0, dev->stream>>>(
      s, seg, (__half*)p16, rows, T, H > 0 ? H : 1, scale, fill_block);
  return vkg_check_launch("attn_softmax");
}

extern "C" int vkg_attn_softmax_bwd(vkg_device* dev, const float* dp, const void* p16, void* ds16,
                                    int64_t rows, int T, float scale, int fill_block) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dp && p16 && ds16 && rows > 0 && T > 0, "attn_softmax_bwd: bad arguments");
  const int wpb = 8;
  if (T <= 1024 && rows % T == 0 && rows / T < (1ll << 31)) {
#define VKG_SM(NV)                                                                                          \
  VKG_RUN(VKG_K_SMALL, rows * T <= SHORT_ELEMS, k_attn_softmax_bwd_reg<NV>,                                 \
          dim3((unsigned)(rows / T), (unsigned)((T + 7) / 8)), 256, dp, (const __half*)p16, (__half*)ds16,  \
          T, scale, fill_block)
    if (T <= 128) VKG_SM(4);
    else if (T <= 256) VKG_SM(8);
    else if (T <= 512) VKG_SM(16);
    else VKG_SM(32);
#undef VKG_SM
    return vkg_check_launch("attn_softmax_bwd");
  }
  k_attn_softmax_bwd<<<(unsigned)((rows + wpb - 1) / wpb), wpb * 32, 0, dev->stream>>>(
      dp, (const __half*)p16, (__half*)ds16, rows, T, scale, fill_block);
  return vkg_check_launch("attn_softmax_bwd");
}

extern "C" int vkg_split_qkv(vkg_device* dev, const float* qkv, const float* bias, void* q16,
                             void* k16, void* v16, int64_t n, int D, int T, int H, int hd) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(qkv && bias && q16 && k16 && v16 && n > 0, "split_qkv: bad arguments");
  int rows;
  dim3 grid;
  if (heads_v4(n, D, T, H, hd, 3, &rows, &grid) && aligned16(qkv, bias) &&
      (((uintptr_t)q16 | (uintptr_t)k16 | (uintptr_t)v16) & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_heads_v4<PERM_SPLIT_QKV>, grid, TPB, qkv, bias, nullptr, (__half*)q16,
            (__half*)k16, (__half*)v16, rows, D, T, H, hd);
    return vkg_check_launch("split_qkv");
  }
  k_split_qkv<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(qkv, bias, (__half*)q16, (__half*)k16,
                                                          (__half*)v16, n, D, T, H, hd);
  return vkg_check_launch("split_qkv");
}

extern "C" int vkg_merge_qkv_grad(vkg_device* dev, const float* dq, const float* dk, const float* dv,
                                  void* dqkv16, int64_t n, int D, int T, int H, int hd) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dq && dk && dv && dqkv16 && n > 0, "merge_qkv_grad: bad arguments");
  int rows;
  dim3 grid;
  if (heads_v4(n, D, T, H, hd, 3, &rows, &grid) && aligned16(dq, dk, dv) && ((uintptr_t)dqkv16 & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_heads_v4<PERM_MERGE_QKV>, grid, TPB, dq, dk, dv, (__half*)dqkv16, nullptr,
            nullptr, rows, D, T, H, hd);
    return vkg_check_launch("merge_qkv_grad");
  }
  k_merge_qkv_grad<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(dq, dk, dv, (__half*)dqkv16, n, D, T,
                                                               H, hd);
  return vkg_check_launch("merge_qkv_grad");
}

extern "C" int vkg_merge_heads(vkg_device* dev, const float* src, void* y16, int64_t n, int D, int T,
                               int H, int hd) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(src && y16 && n > 0, "merge_heads: bad arguments");
  int rows;
  dim3 grid;
  if (heads_v4(n, D, T, H, hd, 1, &rows, &grid) && aligned16(src) && ((uintptr_t)y16 & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_heads_v4<PERM_MERGE>, grid, TPB, src, nullptr, nullptr, (__half*)y16,
            nullptr, nullptr, rows, D, T, H, hd);
    return vkg_check_launch("merge_heads");
  }
  k_merge_heads<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(src, (__half*)y16, n, D, T, H, hd);
  return vkg_check_launch("merge_heads");
}

extern "C" int vkg_split_heads(vkg_device* dev, const float* src, void* dst16, int64_t n, int D,
                               int T, int H, int hd) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(src && dst16 && n > 0, "split_heads: bad arguments");
  int rows;
  dim3 grid;
  if (heads_v4(n, D, T, H, hd, 1, &rows, &grid) && aligned16(src) && ((uintptr_t)dst16 & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_heads_v4<PERM_SPLIT>, grid, TPB, src, nullptr, nullptr, (__half*)dst16,
            nullptr, nullptr, rows, D, T, H, hd);
    return vkg_check_launch("split_heads");
  }
  k_split_heads<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(src, (__half*)dst16, n, D, T, H, hd);
  return vkg_check_launch("split_heads");
}

extern "C" int vkg_embed(vkg_device* dev, const float* tok, const float* pos, const uint32_t* ids,
                         const uint32_t* seg, float* x, int64_t n, int D, int T) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(tok && pos && ids && x && n > 0, "embed: bad arguments");
  if (D % 4 == 0 && n < (1ll << 31) && ((((uintptr_t)tok | (uintptr_t)pos | (uintptr_t)x) & 15) == 0)) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ROWS, k_embed_v4, dim3(flat_grid(dev, n / 4)), TPB, (const float4*)tok,
            (const float4*)pos, ids, seg, (float4*)x, (int)(n / 4), D / 4, T);
    return vkg_check_launch("embed_v4");
  }
  k_embed<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(tok, pos, ids, seg, x, n, D, T);
  return vkg_check_launch("embed");
}

extern "C" int vkg_gather_rows(vkg_device* dev, const float* src, const uint32_t* rows, float* dst, int n,
                               int D) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(src && rows && dst && n > 0 && D > 0 && D % 4 == 0 &&
                  ((((uintptr_t)src | (uintptr_t)dst) & 15) == 0),
              "gather_rows: D must be a multiple of 4 and the rows 16-byte aligned");
  VKG_RUN(VKG_K_SMALL, (int64_t)n * D <= SHORT_ROWS, k_gather_rows, dim3((unsigned)n), TPB, (const float4*)src, rows,
          (float4*)dst, D / 4);
  return vkg_check_launch("gather_rows");
}

extern "C" int vkg_embed_bwd(vkg_device* dev, const float* dx, const uint32_t* ids,
                             const uint32_t* seg, float* dtok, float* dpos, int64_t n, int D, int T) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dx && ids && dtok && dpos && n > 0, "embed_bwd: bad arguments");
  if (D % 4 == 0 && n < (1ll << 31) && ((((uintptr_t)dx | (uintptr_t)dtok | (uintptr_t)dpos) & 15) == 0)) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ROWS, k_embed_bwd_v4, dim3(flat_grid(dev, n / 4)), TPB, (const float4*)dx, ids,
            seg, (float4*)dtok, (float4*)dpos, (int)(n / 4), D / 4, T);
    return vkg_check_launch("embed_bwd_v4");
  }
  k_embed_bwd<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(dx, ids, seg, dtok, dpos, n, D, T);
  return vkg_check_launch("embed_bwd");
}

extern "C" int64_t vkg_embed_bwd_scratch_bytes(int64_t rows) {
  // keys[2][rows rounded up to 4], next[2][rows], has_prev[2][rows]
  return rows > 0 ? (6 * rows + 8) * (int64_t)sizeof(int) : 0;
}

extern "C" int vkg_embed_bwd_det(vkg_device* dev, const float* dx, const uint32_t* ids,
                                 const uint32_t* seg, float* dtok, float* dpos, void* scratch,
                                 int64_t n, int D, int T) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(dx && ids && dtok && dpos && scratch && n > 0 && D > 0 && T > 0,
              "embed_bwd_det: bad arguments");
  VKG_REQUIRE(D % 4 == 0 && D <= 1024 && n % D == 0 && n / D < (1ll << 30) &&
                  ((((uintptr_t)dx | (uintptr_t)dtok | (uintptr_t)dpos | (uintptr_t)scratch) & 15) == 0),
              "embed_bwd_det: D must be a multiple of 4 up to 1024 and the tables 16-byte aligned "
              "(use vkg_embed_bwd otherwise)");
  const int rows = (int)(n / D), rows_p = (rows + 3) & ~3;
  int* keys = static_cast<int*>(scratch);
  int* next = keys + 2 * (size_t)rows_p;
  int* has_prev = next + 2 * (size_t)rows;
  VKG_RUN(VKG_K_SMALL, n <= SHORT_ROWS, k_embed_keys, dim3((unsigned)((2 * rows_p + 255) / 256)), 256, ids, seg,
          keys, has_prev, rows, rows_p, T);
  if (vkg_check_launch("embed_keys")) return 1;
  VKG_RUN(VKG_K_SMALL, n <= SHORT_ROWS, k_embed_chain, dim3((unsigned)((2 * rows + 7) / 8)), 256, keys, next,
          has_prev, rows, rows_p);
  if (vkg_check_launch("embed_chain")) return 1;
  const dim3 grid((unsigned)((rows + 7) / 8), 2);
#define VKG_EB(NV)                                                                            \
  VKG_RUN(VKG_K_SMALL, n <= SHORT_ROWS, k_embed_bwd_chain<NV>, grid, 256, dx, ids, seg, next, \
          has_prev, dtok, dpos, rows, D, T)
  switch ((D + 127) / 128) {
    case 1: VKG_EB(1); break;
    case 2: VKG_EB(2); break;
    case 3: VKG_EB(3); break;
    case 4: VKG_EB(4); break;
    case 5: VKG_EB(5); break;
    case 6: VKG_EB(6); break;
    case 7: VKG_EB(7); break;
    default: VKG_EB(8); break;
  }
#undef VKG_EB
  return vkg_check_launch("embed_bwd_chain");
}

extern "C" int vkg_residual(vkg_device* dev, const float* acc, const float* bias, const float* res,
                            float* out, int64_t n, int D) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(acc && bias && res && out && n > 0, "residual: bad arguments");
  int nrow;
  dim3 grid;
  if (D > 0 && rows_v4(n, D, &nrow, &grid) && aligned16(acc, bias, res, out)) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_rows_v4<V4_RESIDUAL>, grid, TPB, (const float4*)acc, (const float4*)bias,
            (const float4*)res, (float4*)out, nullptr, nrow, D / 4, 0);
    return vkg_check_launch("residual");
  }
  k_residual<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(acc, bias, res, out, n, D);
  return vkg_check_launch("residual");
}

extern "C" int vkg_add(vkg_device* dev, const float* a, const float* b, float* out, void* out16,
                       int64_t n) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(a && b && (out || out16) && n > 0, "add: bad arguments");
  // in place (out == a or b) is fine: a thread reads a value before it writes it
  if (n % 4 == 0 && aligned16(a, b, out) && ((uintptr_t)out16 & 7) == 0) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_flat_v4<V4_ADD>, dim3(flat_grid(dev, n / 8)), TPB, (const float4*)a,
            (const float4*)b, (float4*)out, (uint2*)out16, n / 4, 0);
    return vkg_check_launch("add");
  }
  k_add<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(a, b, out, (__half*)out16, n);
  return vkg_check_launch("add");
}

extern "C" int vkg_add_bias(vkg_device* dev, float* x, const float* bias, int64_t n, int ncol) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(x && bias && n > 0 && ncol > 0, "add_bias: bad arguments");
  int nrow;
  dim3 grid;
  if (rows_v4(n, ncol, &nrow, &grid) && aligned16(x, bias)) {
    VKG_RUN(VKG_K_SMALL, n <= SHORT_ELEMS, k_rows_v4<V4_ADD_BIAS>, grid, TPB, (const float4*)x, (const float4*)bias,
            nullptr, (float4*)x, nullptr, nrow, ncol / 4, 0);
    return vkg_check_launch("add_bias");
  }
  k_add_bias<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(x, bias, n, ncol);
  return vkg_check_launch("add_bias");
}

extern "C" int vkg_grad_add(vkg_device* dev, const float* g, float* arena, int64_t n, int64_t off) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(g && arena && n > 0 && off >= 0, "grad_add: bad arguments");
  k_grad_add<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(g, arena + off, n);
  return vkg_check_launch("grad_add");
}

extern "C" int vkg_grad_pull(vkg_device* dev, const float* arena, float* g, int64_t n, int64_t off,
                             float scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(g && arena && n > 0 && off >= 0, "grad_pull: bad arguments");
  k_grad_pull<<<flat_grid(dev, n), TPB, 0, dev->stream>>>(arena + off, g, n, scale);
  return vkg_check_launch("grad_pull");
}

extern "C" int vkg_bucket_pack16(vkg_device* dev, const float* src, void* dst16, int dtype, int64_t n,
                                 float scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(src && dst16 && n > 0, "bucket_pack16: bad arguments");
  if (dtype == VKG_F16)
    k_pack16<__half><<<flat_grid(dev, n), TPB, 0, dev->stream>>>(src, (__half*)dst16, n, scale);
  else if (dtype == VKG_BF16)
    k_pack16<__nv_bfloat16><<<flat_grid(dev, n), TPB, 0, dev->stream>>>(src, (__nv_bfloat16*)dst16, n,
                                                                         scale);
  else
    VKG_FAIL("bucket_pack16: dtype must be f16 or bf16");
  return vkg_check_launch("bucket_pack16");
}

extern "C" int vkg_bucket_unpack16(vkg_device* dev, const void* src16, int dtype, float* dst,
                                   int64_t n, float scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(src16 && dst && n > 0, "bucket_unpack16: bad arguments");
  if (dtype == VKG_F16)
    k_unpack16<__half><<<flat_grid(dev, n), TPB, 0, dev->stream>>>((const __half*)src16, dst, n, scale);
  else if (dtype == VKG_BF16)
    k_unpack16<__nv_bfloat16><<<flat_grid(dev, n), TPB, 0, dev->stream>>>((const __nv_bfloat16*)src16,
                                                                           dst, n, scale);
  else
    VKG_FAIL("bucket_unpack16: dtype must be f16 or bf16");
  return vkg_check_launch("bucket_unpack16");
}
