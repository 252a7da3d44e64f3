// The GEMM trio (Y = X W, dX = dY W^T, dW = X^T dY) and its batched form for
// sm_100a: TMA -> 128B-swizzled shared memory ring -> tcgen05.mma issued by one
// thread -> fp32 accumulators in TMEM (two stages, so the epilogue of tile i
// overlaps the main loop of tile i+1) -> tcgen05.ld epilogue with the fused
// bias / activation / activation-derivative / residual / narrowing.
//
// One persistent CTA per SM, 576 threads:
//   warp 0       TMA producer (one lane; of a CTA pair: converged, one elected lane per stage)
//   warp 1       TMEM allocation + MMA issue (converged, one elected lane per instruction)
//   warps 2..17  epilogue; warp w reads TMEM lanes 32*(w%4) .. +31 and takes every
//                fourth 16-column chunk.  The epilogue is instruction-issue / latency
//                bound, so it gets four warps per scheduler and a compile-time mask.
//
// Transposed operands are never materialised (the reference makes the same
// point for its cooperative-matrix loads, kernels.py:45-49): "A stored K x M"
// and "B stored K x N" are loaded as MN-major tiles and the shared-memory /
// instruction descriptors say so.
//
// Two kernels share the role code: gemm_tcgen05_kernel (128 x {64..256} tiles, one CTA
// each) and gemm_cta_pair_kernel (256 x {192, 256} tiles on 2-CTA clusters with
// tcgen05.mma.cta_group::2, each CTA loading its rows of A and half of the B tile); the host
// chooses between them, and the width, from a fitted time model (choose_tiles).
//
// Every mbarrier wait is bounded by a clock64 budget; a wait that gives up
// sets an error word the host reads at the next synchronisation, the CTA
// stops issuing work, frees its TMEM and returns.
#include "common.cuh"
#include "tcgen05.cuh"

#include <algorithm>
#include <string>
#include <unordered_map>

namespace {

using namespace tc05;

constexpr int BM = 128;            // rows of C per tile = UMMA M
constexpr int BK = 64;             // K elements per k-block = 128 bytes of f16 = one swizzle row
constexpr int UMMA_K = 16;         // K per tcgen05.mma.kind::f16
constexpr int A_STAGE_BYTES = BM * BK * 2;
constexpr int MAX_STAGES = 8;
constexpr int EPI_WARPS = 16;      // four per TMEM lane quarter, each takes every fourth 16-column chunk
constexpr int NUM_THREADS = (2 + EPI_WARPS) * 32;
constexpr int TMEM_COLS = 512;     // whole TMEM: two 256-column accumulators
constexpr int ACC_COLS = 256;
constexpr int RING_BYTES = 196608; // shared-memory ring budget
constexpr int EPI_STAGE_BYTES = 32 * 16 * 4;  // one 32x16 fp32 chunk per epilogue warp (XOR-swizzled)
constexpr int SMEM_BYTES = RING_BYTES + EPI_WARPS * EPI_STAGE_BYTES + 1024 /*align slack*/ +
                           256 /*barriers*/;
constexpr int GROUP_M = 8;         // m-tiles per rasterisation band

struct GemmParams {
  int M, N, K;
  int nb0, nb1;
  int tiles_m, tiles_n;
  int bn, stage_kb, num_kb;
  int split_k, kb_per_split;   // split_k > 1: z1 is the K slice, not a batch index
  int causal;                  // 0 none, 1 skip tiles above the diagonal, 2/3 clip the K range
  int a_mn, b_mn;              // MN-major, and wide (Feed): OP_MN | OP_WIDE
  uint32_t idesc;
  int c_dtype, act, dact, vec_ok;
  long long ldc, sC0, sC1;
  void* C;
  void* C2;
  const float* bias;
  float* pre;
  const float* dact_z;
  const float* residual;
  float* colsum;               // optional: [4 * row blocks][N] partial column sums of the output
  float alpha;
  int tma_store;               // epilogue stores C (and pre) through tensor maps
  uint32_t* err;
};

enum : int { OP_MN = 1, OP_WIDE = 2 };

// The ring of one CTA.
struct RingShape {
  int stage_bytes, stages;
  __host__ __device__ RingShape(bool pair, int bn, bool b_mn, int stage_kb) {
    // rows of a K-major B, or columns of an MN-major one, which are loaded in whole groups of 64 (a 96-column
    // half of a pair's tile loads two and uses one and a half)
    const int rows_b = pair ? bn / 2 : bn;
    stage_bytes = stage_kb * (A_STAGE_BYTES + (b_mn ? (rows_b + 63) / 64 * 64 : rows_b) * 128);
    stages = RING_BYTES / stage_bytes < MAX_STAGES ? RING_BYTES / stage_bytes : MAX_STAGES;
  }
};

struct TileCoord {
  int z0, z1, m0, n0;
};

// bm: rows of C per tile (BM, or 2 * BM for a CTA pair); m_off: this CTA's rows inside it.
__device__ __forceinline__ TileCoord tile_coord(const GemmParams& p, int t, int bm = BM, int m_off = 0) {
  int per_batch = p.tiles_m * p.tiles_n;
  int z = t / per_batch;
  int r = t - z * per_batch;
  int band = GROUP_M * p.tiles_n;
  int g = r / band;
  int first_m = g * GROUP_M;
  int gsize = min(p.tiles_m - first_m, GROUP_M);
  int in_band = r - g * band;
  TileCoord c;
  c.m0 = (first_m + in_band % gsize) * bm + m_off;
  c.n0 = (in_band / gsize) * p.bn;
  c.z0 = z % p.nb0;
  c.z1 = z / p.nb0;
  return c;
}

// K-block range of a work unit: everything, slice z1 when K is split, or the part of K
// a causal operand is non-zero in.  nkb == 0 means the tile is skipped by every role.
__device__ __forceinline__ void kb_range(const GemmParams& p, const TileCoord& c, int& kb0, int& nkb) {
  if (p.split_k > 1) {
    kb0 = c.z1 * p.kb_per_split;
    nkb = min(p.kb_per_split, p.num_kb - kb0);
  } else {
    kb0 = 0;
    nkb = p.num_kb;
    if (p.causal == 1) {
      if (c.n0 > c.m0 + BM - 1) nkb = 0;                  // wholly above the diagonal
    } else if (p.causal == 2) {
      nkb = min(p.num_kb, (c.m0 + BM + BK - 1) / BK);    // A[m, k] = 0 for k > m
    } else if (p.causal == 3) {
      kb0 = c.m0 / BK;                                    // A^T[k, m] = 0 for k < m
      nkb = p.num_kb - kb0;
    }
  }
}

// Compile-time epilogue feature mask.  E_GENERIC reads every flag (and the vector
// alignment flag) at run time; the specialised masks assume 16-byte aligned operands.
enum : int {
  E_BIAS = 1, E_PRE = 2, E_ACT = 4, E_DACT = 8, E_RES = 16, E_C2 = 32, E_F16 = 64, E_BF16 = 128,
  E_COLSUM = 256,
  E_GENERIC = 1 << 20
};

template <typename T2, typename T>
__device__ __forceinline__ void store4_16(T* c, const float* v, bool vec);

template <>
__device__ __forceinline__ void store4_16<__half2, __half>(__half* c, const float* v, bool vec) {
  if (vec) {
    __half2 h[2] = {__floats2half2_rn(v[0], v[1]), __floats2half2_rn(v[2], v[3])};
    *reinterpret_cast<uint2*>(c) = *reinterpret_cast<uint2*>(h);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = __float2half_rn(v[j]);
  }
}

template <>
__device__ __forceinline__ void store4_16<__nv_bfloat162, __nv_bfloat16>(__nv_bfloat16* c,
                                                                         const float* v, bool vec) {
  if (vec) {
    __nv_bfloat162 h[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
    *reinterpret_cast<uint2*>(c) = *reinterpret_cast<uint2*>(h);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = __float2bfloat16_rn(v[j]);
  }
}

__device__ __forceinline__ float4 ld4(const float* p, long long off, bool vec) {
  if (vec) return *reinterpret_cast<const float4*>(p + off);
  return make_float4(p[off], p[off + 1], p[off + 2], p[off + 3]);
}

__device__ __forceinline__ void st4(float* p, long long off, float4 v, bool vec) {
  if (vec) {
    *reinterpret_cast<float4*>(p + off) = v;
  } else {
    p[off] = v.x; p[off + 1] = v.y; p[off + 2] = v.z; p[off + 3] = v.w;
  }
}

// Operand of the epilogue that is read per element (the saved pre-activation, or the residual):
// requested one chunk ahead, so that its trip to memory (0.7 us per chunk, more than the rest of a
// chunk together) lies under the wait for the accumulator and the arithmetic of the chunk before.
template <int MODE>
__device__ __forceinline__ void epilogue_fetch(const GemmParams& p, float4 (&extra)[4],
                                               const long long off0, const long long step, unsigned ok) {
  if (!(MODE & (E_DACT | E_RES)) || (MODE & E_GENERIC)) return;
  const float* from = (MODE & E_DACT) ? p.dact_z : p.residual;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    extra[i] = (ok >> i) & 1u ? ld4(from, off0 + i * step, true) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// One lane's share of a 32x16 chunk through the fused epilogue: four rows (8*i +
// sub_row), four consecutive columns each.  In this layout four lanes cover the 16
// columns (64 bytes) of one row, so every global access of the warp is eight
// row-contiguous 64-byte pieces.  All loads of one kind are issued before the first
// dependent use: C may alias the inputs as far as the compiler knows, so a
// load-compute-store loop would serialise eight memory round trips.
//
// lanes: the lanes of the warp that call this together (those whose columns exist).
// cs_row: which row of p.colsum this warp's 32 rows add up into.  The sums are taken over
// the values as stored (after the narrowing), rows in a fixed order: lanes first add their
// four rows, then the eight row groups are folded by shuffles.
template <int MODE>
__device__ __forceinline__ void epilogue_chunk(const GemmParams& p, float4 (&v)[4], float4 (&extra)[4],
                                               const long long off0, const long long step, unsigned ok, int col,
                                               int cs_row, unsigned lanes) {
  static_assert((MODE & E_GENERIC) || (MODE & (E_DACT | E_RES)) != (E_DACT | E_RES), "one fetched operand");
  constexpr bool G = (MODE & E_GENERIC) != 0;
  const bool has_colsum = G ? (p.colsum != nullptr) : (MODE & E_COLSUM) != 0;
  const bool vec = G ? (p.vec_ok != 0) : true;
  const bool has_bias = G ? (p.bias != nullptr) : (MODE & E_BIAS) != 0;
  const bool has_pre = G ? (p.pre != nullptr) : (MODE & E_PRE) != 0;
  const bool has_act = G ? (p.act != 0) : (MODE & E_ACT) != 0;
  const bool has_dact = G ? (p.dact_z != nullptr) : (MODE & E_DACT) != 0;
  const bool has_res = G ? (p.residual != nullptr) : (MODE & E_RES) != 0;
  const bool has_c2 = G ? (p.C2 != nullptr) : (MODE & E_C2) != 0;
  const int c_dtype = G ? p.c_dtype : ((MODE & E_F16) ? VKG_F16 : (MODE & E_BF16) ? VKG_BF16 : VKG_F32);
  if (G && has_dact) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      extra[i] = (ok >> i) & 1u ? ld4(p.dact_z, off0 + i * step, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float4 b = make_float4(0.f, 0.f, 0.f, 0.f);
  if (has_bias) b = ld4(p.bias, col, vec);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i].x = v[i].x * p.alpha + b.x; v[i].y = v[i].y * p.alpha + b.y;
    v[i].z = v[i].z * p.alpha + b.z; v[i].w = v[i].w * p.alpha + b.w;
  }
  if (has_pre) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((ok >> i) & 1u) st4(p.pre, off0 + i * step, v[i], vec);
  }
  // the kind of activation is tested once per chunk, not per element
  if (has_act) {
    if (p.act == VKG_ACT_GELU) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i].x = vkg_gelu(v[i].x); v[i].y = vkg_gelu(v[i].y);
        v[i].z = vkg_gelu(v[i].z); v[i].w = vkg_gelu(v[i].w);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i].x = vkg_act(v[i].x, p.act); v[i].y = vkg_act(v[i].y, p.act);
        v[i].z = vkg_act(v[i].z, p.act); v[i].w = vkg_act(v[i].w, p.act);
      }
    }
  }
  if (has_dact) {
    if (p.dact == VKG_ACT_GELU) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i].x *= vkg_dgelu(extra[i].x); v[i].y *= vkg_dgelu(extra[i].y);
        v[i].z *= vkg_dgelu(extra[i].z); v[i].w *= vkg_dgelu(extra[i].w);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i].x *= vkg_dact(extra[i].x, p.dact); v[i].y *= vkg_dact(extra[i].y, p.dact);
        v[i].z *= vkg_dact(extra[i].z, p.dact); v[i].w *= vkg_dact(extra[i].w, p.dact);
      }
    }
  }
  if (has_res) {
    if (G) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        extra[i] = (ok >> i) & 1u ? ld4(p.residual, off0 + i * step, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i].x += extra[i].x; v[i].y += extra[i].y; v[i].z += extra[i].z; v[i].w += extra[i].w;
    }
  }
  // narrowed once: the column sums are of the values as stored
  uint2 h[4];
  if (c_dtype == VKG_F16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __half2 a = __floats2half2_rn(v[i].x, v[i].y), b = __floats2half2_rn(v[i].z, v[i].w);
      h[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
  }
  if (has_colsum) {
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (!((ok >> i) & 1u)) continue;
      float4 t = v[i];
      if (c_dtype == VKG_F16) {
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&h[i].x));
        const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&h[i].y));
        t = make_float4(lo.x, lo.y, hi.x, hi.y);
      } else if (c_dtype == VKG_BF16) {
        t.x = __bfloat162float(__float2bfloat16_rn(t.x)); t.y = __bfloat162float(__float2bfloat16_rn(t.y));
        t.z = __bfloat162float(__float2bfloat16_rn(t.z)); t.w = __bfloat162float(__float2bfloat16_rn(t.w));
      }
      s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
    }
#pragma unroll
    for (int d = 4; d < 32; d <<= 1) {
      s.x += __shfl_xor_sync(lanes, s.x, d);
      s.y += __shfl_xor_sync(lanes, s.y, d);
      s.z += __shfl_xor_sync(lanes, s.z, d);
      s.w += __shfl_xor_sync(lanes, s.w, d);
    }
    if ((threadIdx.x & 31) < 4) st4(p.colsum, (long long)cs_row * p.N + col, s, vec);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (!((ok >> i) & 1u)) continue;
    const float f[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
    if (c_dtype == VKG_F32) {
      st4(reinterpret_cast<float*>(p.C), off0 + i * step, v[i], vec);
    } else if (c_dtype == VKG_F16) {
      __half* c = reinterpret_cast<__half*>(p.C) + off0 + i * step;
      if (vec) *reinterpret_cast<uint2*>(c) = h[i];
      else store4_16<__half2, __half>(c, f, false);
    } else {
      store4_16<__nv_bfloat162, __nv_bfloat16>(reinterpret_cast<__nv_bfloat16*>(p.C) + off0 + i * step, f, vec);
    }
    if (has_c2) {
      __half* c = reinterpret_cast<__half*>(p.C2) + off0 + i * step;
      store4_16<__half2, __half>(c, f, vec);
    }
  }
}

// Epilogues that only WRITE (plain, bias, bias + keep z + activation, narrowing) can leave the
// transposition to the TMA: the warp keeps the TMEM layout (lane = row, 16 columns), applies
// the fused arithmetic in registers, writes its 32 x 16 chunk into the staging area in the
// hardware's swizzled layout and one lane issues a tensor-map store of the box.  Compared
// with the per-lane path this drops the shared-memory read-back, the address arithmetic, the
// predicates (the box is clipped at the tensor's edge) and the global store instructions.
constexpr int E_NO_TMA = E_DACT | E_RES | E_C2 | E_COLSUM | E_GENERIC;

// 32 x 16 fp32: 64-byte rows, 16-byte piece j of row r at ((j ^ ((r >> 1) & 3)) << 4) -- the
// 64-byte swizzle of the tensor map, and conflict-free for one-row-per-lane writes.
__device__ __forceinline__ void stage_chunk_f32(const float (&v)[16], uint8_t* stage, int lane) {
#pragma unroll
  for (int j = 0; j < 4; ++j)
    *reinterpret_cast<float4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) =
        make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}

// 32 x 16 halves: 32-byte rows, piece j of row r at ((j ^ ((r >> 2) & 1)) << 4) (32-byte swizzle)
template <bool BF>
__device__ __forceinline__ void stage_chunk_16(const float (&v)[16], uint8_t* stage, int lane) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    uint4 pk;
    uint32_t* w = reinterpret_cast<uint32_t*>(&pk);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (BF) {
        __nv_bfloat162 h = __floats2bfloat162_rn(v[8 * j + 2 * e], v[8 * j + 2 * e + 1]);
        w[e] = *reinterpret_cast<uint32_t*>(&h);
      } else {
        __half2 h = __floats2half2_rn(v[8 * j + 2 * e], v[8 * j + 2 * e + 1]);
        w[e] = *reinterpret_cast<uint32_t*>(&h);
      }
    }
    *reinterpret_cast<uint4*>(stage + lane * 32 + ((j ^ ((lane >> 2) & 1)) << 4)) = pk;
  }
}

// NC 32 x 16 chunks (rows row0.., columns col0.., col1..) through the write-only epilogue, in the
// warp's 2 KB of staging: one fp32 chunk, or two 16-bit ones, which are then filled, fenced and
// handed to the TMA together -- one wait for tensor memory, one proxy fence and one bulk
// async-group for both (a chunk on its own is 700 cycles of latencies in a row).  The staging is
// filled again once the last store has been read (bulk async-groups belong to the issuing thread,
// so lane 0 waits and the warp meets it); twice the staging at the cost of a ring stage measured
// no better.
template <int MODE, int NC>
__device__ __forceinline__ void epilogue_chunks_tma(const GemmParams& p, const CUtensorMap* tmC,
                                                    const CUtensorMap* tmP, uint32_t (&r)[NC][16],
                                                    uint8_t* stage, int lane, int col0, int col1, int row0,
                                                    int z0, int z1) {
  static_assert(NC == 1 || ((MODE & (E_F16 | E_BF16)) && !(MODE & E_PRE)), "two chunks only where both fit");
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int col = c ? col1 : col0;
    float v[16];
    if (MODE & E_BIAS) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        // N is a multiple of 8, the chunk may reach 8 past it
        const float4 b = col + 4 * g < p.N ? *reinterpret_cast<const float4*>(p.bias + col + 4 * g)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * g] = fmaf(__uint_as_float(r[c][4 * g]), p.alpha, b.x);
        v[4 * g + 1] = fmaf(__uint_as_float(r[c][4 * g + 1]), p.alpha, b.y);
        v[4 * g + 2] = fmaf(__uint_as_float(r[c][4 * g + 2]), p.alpha, b.z);
        v[4 * g + 3] = fmaf(__uint_as_float(r[c][4 * g + 3]), p.alpha, b.w);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[c][j]) * p.alpha;
    }
    if (c == 0) {
      if (lane == 0) bulk_wait_read_all();
      __syncwarp();
    }
    if (MODE & E_PRE) {
      stage_chunk_f32(v, stage, lane);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        tma_store_4d(tmP, smem_u32(stage), col, row0, z0, z1);
        bulk_commit_group();
      }
    }
    if (MODE & E_ACT) {
      if (p.act == VKG_ACT_GELU) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = vkg_gelu(v[j]);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = vkg_act(v[j], p.act);
      }
    }
    if (MODE & E_PRE) {
      if (lane == 0) bulk_wait_read_all();
      __syncwarp();
    }
    uint8_t* to = stage + c * (EPI_STAGE_BYTES / 2);
    if (MODE & E_F16) stage_chunk_16<false>(v, to, lane);
    else if (MODE & E_BF16) stage_chunk_16<true>(v, to, lane);
    else stage_chunk_f32(v, to, lane);
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    tma_store_4d(tmC, smem_u32(stage), col0, row0, z0, z1);
    if (NC == 2) tma_store_4d(tmC, smem_u32(stage + EPI_STAGE_BYTES / 2), col1, row0, z0, z1);
    bulk_commit_group();
  }
}

// Per-CTA constants shared by the three roles.
struct CtaCtx {
  uint32_t base, stage_bytes, full0, empty0, tfull0, tempty0, tmem_base;
  int n_stages;
  volatile uint32_t* abort_flag;
  uint8_t* epi_stage;
};

// Position in the ring.  A stage's first fill waits for nobody.
struct Ring {
  int stage = 0;
  uint32_t phase = 0;
  bool wrapped = false;
  __device__ __forceinline__ void step(int n_stages) {
    if (++stage == n_stages) {
      stage = 0;
      phase ^= 1u;
      wrapped = true;
    }
  }
};

// How an operand comes into the ring.  What a k-block of a narrow tile costs is neither bytes nor tensor
// time but the instructions around them: 115 cycles for a wait, 50 to 100 for each load, in the loop of
// the warp that loads and again in the loop of the warp that multiplies.  With one k-block to a stage
// and a load for every 64 columns both loops took 383 (NT) to 490 (TN) cycles where the tensor core needs
// 192.  So a stage may hold two k-blocks (stage_kb_for), and an operand whose
// contiguous dimension is whole 64-element pieces is wide: its map splits that dimension in two, and one
// load brings the stage's pieces, each a tile of its own ([k-block][row][64] of a K-major operand,
// [64 columns][k][64] of an MN-major one).  Others take a load per piece, into the same places.
// 1024 x 768 x 3072 (NN, residual): 15.4 -> 11.7 us, 768 x 2304 x 1024 (TN) 9.1 -> 7.6.
struct Feed {
  int c0, c1, c2;        // map coordinates; a load per piece moves c0 on by 64
  int s0, s1, s2;        // their step per stage
  int loads;
  uint32_t step;         // shared-memory bytes from one load to the next
  __device__ __forceinline__ Feed(int kind, int kb0, int at, int rows, int stage_kb) {
    const bool mn = (kind & OP_MN) != 0, wide = (kind & OP_WIDE) != 0;
    c0 = wide ? 0 : mn ? at : kb0 * BK;
    c1 = mn ? kb0 * BK : at;
    c2 = !wide ? 0 : mn ? at / 64 : kb0;
    s0 = wide || mn ? 0 : stage_kb * BK;
    s1 = mn ? stage_kb * BK : 0;
    s2 = wide && !mn ? stage_kb : 0;
    loads = wide ? 1 : mn ? (rows + 63) / 64 : stage_kb;
    step = mn ? (uint32_t)stage_kb * 8192u : (uint32_t)rows * 128u;
  }
  template <bool PAIR>
  __device__ __forceinline__ void load(uint32_t dst, const CUtensorMap* map, uint32_t bar, const TileCoord& tc) {
    int x = c0;
    for (int i = loads;;) {
      if (PAIR) tma_load_5d_pair(dst, map, bar, x, c1, c2, tc.z0, tc.z1);
      else tma_load_5d(dst, map, bar, x, c1, c2, tc.z0, tc.z1);
      if (--i == 0) break;
      x += 64;
      dst += step;
    }
  }
  __device__ __forceinline__ void next() {
    c0 += s0;
    c1 += s1;
    c2 += s2;
  }
};

// TMA producer of a single CTA (one lane) or of one CTA of a pair (the whole warp): stream the k-blocks of a
// work unit's operands into the ring.  b_at: the CTA's first column of B.
// A load issued from a branch that only lane 0 takes has its operands moved from vector registers one by
// one.  Where a k-block of a 256-column pair tile comes in four loads, that paces the tile (2544 x 1392 x 3640
// TN: 26.4 us, 24.0 with an elected lane of a converged warp).  A single CTA's short tiles start 0.05 to 0.1 us
// later that way (280 x 832 x 264: 7.08 -> 7.21), and gain nothing.
template <bool PAIR>
__device__ __forceinline__ bool produce(const CtaCtx& cx, const GemmParams& p, const CUtensorMap* tmA,
                                        const CUtensorMap* tmB, TileCoord tc, int b_at, uint32_t rank, Ring& at) {
  int kb0, nkb;
  kb_range(p, tc, kb0, nkb);
  if (p.split_k > 1) tc.z1 = 0;   // operands are not batched along the slice index
  Feed a(p.a_mn, kb0, tc.m0, BM, p.stage_kb), b(p.b_mn, kb0, b_at, PAIR ? p.bn / 2 : p.bn, p.stage_kb);
  const uint32_t a_bytes = (uint32_t)p.stage_kb * A_STAGE_BYTES;
  for (int kb = 0; kb < nkb; kb += p.stage_kb) {
    // (one expression for both kinds of wait made a single CTA's launches 0.03 us longer)
    if (PAIR) {
      if (at.wrapped &&
          !mbar_wait_warp(cx.empty0 + 8 * at.stage, at.phase ^ 1u, cx.abort_flag, p.err, 0x100u + at.stage))
        return false;
    } else {
      if (at.wrapped && !mbar_wait(cx.empty0 + 8 * at.stage, at.phase ^ 1u, cx.abort_flag, p.err, 0x100u + at.stage))
        return false;
    }
    uint32_t fb = cx.full0 + 8 * at.stage;
    const uint32_t sa = cx.base + at.stage * cx.stage_bytes;
    if (!PAIR || elect_one()) {
      if (PAIR) {
        if (rank == 0) mbar_expect_tx(fb, 2 * cx.stage_bytes);
        fb = mapa_shared(fb, 0);
      } else {
        mbar_expect_tx(fb, cx.stage_bytes);
      }
      a.load<PAIR>(sa, tmA, fb, tc);
      b.load<PAIR>(sa + a_bytes, tmB, fb, tc);
    }
    a.next();
    b.next();
    at.step(cx.n_stages);
  }
  return true;
}

// MMA issue (the whole warp, converged; one elected lane issues each instruction) of a single CTA, or of
// the even-ranked CTA for a pair: accumulate a work unit's k-blocks into one of the two TMEM
// accumulators.  Descriptor halves step along K by 16 elements: 32 bytes further along the 128-byte row
// for a K-major operand, two 8-row groups (2 x 1024 bytes) further down for an MN-major one, whose 64-column
// groups lie a stage's k apart.  All in units of 16 bytes.
template <bool PAIR, int STAGE_KB>
__device__ __forceinline__ bool multiply(const CtaCtx& cx, const GemmParams& p, uint32_t d_tmem, int nkb, Ring& at) {
  const uint32_t d_hi = smem_desc_hi(1024);
  const bool a_mn = (p.a_mn & OP_MN) != 0, b_mn = (p.b_mn & OP_MN) != 0;
  const uint32_t a_lo0 = smem_desc_lo(cx.base, a_mn ? STAGE_KB * 8192 : 16);
  const uint32_t b_lo0 = smem_desc_lo(cx.base + STAGE_KB * A_STAGE_BYTES, b_mn ? STAGE_KB * 8192 : 16);
  const uint32_t a_step = a_mn ? 128u : 2u, b_step = b_mn ? 128u : 2u;
  const uint32_t a_kb = a_mn ? 512u : BM * 8u, b_kb = b_mn ? 512u : (uint32_t)(PAIR ? p.bn / 2 : p.bn) * 8u;
  const uint32_t stage16 = cx.stage_bytes >> 4;
  for (int kb = 0; kb < nkb; kb += STAGE_KB) {
    if (!mbar_wait_warp(cx.full0 + 8 * at.stage, at.phase, cx.abort_flag, p.err, 0x300u + at.stage)) return false;
    tcgen05_fence_after();
    const uint32_t a_lo = a_lo0 + (uint32_t)at.stage * stage16, b_lo = b_lo0 + (uint32_t)at.stage * stage16;
#pragma unroll
    for (int i = 0; i < STAGE_KB; ++i) {
      if (i > 0 && kb + i >= nkb) break;       // the last stage may hold one k-block that does not count
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k) {
        const uint64_t ad = smem_desc_pack(a_lo + i * a_kb + k * a_step, d_hi);
        const uint64_t bd = smem_desc_pack(b_lo + i * b_kb + k * b_step, d_hi);
        if (elect_one()) {
          if (PAIR) umma2_f16(d_tmem, ad, bd, p.idesc, (kb | i | k) != 0 ? 1u : 0u);
          else umma_f16(d_tmem, ad, bd, p.idesc, (kb | i | k) != 0 ? 1u : 0u);
        }
      }
    }
    if (elect_one()) {                         // frees the stage when these MMAs retire
      if (PAIR) umma2_commit(cx.empty0 + 8 * at.stage);
      else umma_commit(cx.empty0 + 8 * at.stage);
    }
    at.step(cx.n_stages);
  }
  return true;
}

template <bool PAIR>
__device__ __forceinline__ bool mma_unit(const CtaCtx& cx, const GemmParams& p, int t, Ring& at, int& acc,
                                         uint32_t& acc_phase) {
  int kb0, nkb;
  kb_range(p, tile_coord(p, t, PAIR ? 2 * BM : BM), kb0, nkb);
  if (nkb <= 0) return true;   // skipped tile: no accumulator, no epilogue
  if (!mbar_wait_warp(cx.tempty0 + 8 * acc, acc_phase ^ 1u, cx.abort_flag, p.err, 0x200u + acc)) return false;
  tcgen05_fence_after();
  const uint32_t d_tmem = cx.tmem_base + (uint32_t)(acc * ACC_COLS);
  // (a kernel for each of the two loops made steps that use both longer: 259 -> 264 us of a block run
  // through the op dictionaries, 2385 -> 2412 of four microbatches with heads of 32)
  if (!(p.stage_kb == 2 ? multiply<PAIR, 2>(cx, p, d_tmem, nkb, at) : multiply<PAIR, 1>(cx, p, d_tmem, nkb, at)))
    return false;
  if (elect_one()) {           // accumulator complete -> epilogue
    if (PAIR) umma2_commit(cx.tfull0 + 8 * acc);
    else umma_commit(cx.tfull0 + 8 * acc);
  }
  acc ^= 1;
  if (acc == 0) acc_phase ^= 1u;
  return true;
}

// Where the lanes of an epilogue warp stand in a 32 x 16 chunk on the per-lane path: four rows
// (8 i + lane / 4) and four columns each.
struct ChunkAt {
  long long off0;      // element offset of the first row; the others follow 8 * ldc apart
  unsigned ok;
};
__device__ __forceinline__ ChunkAt chunk_at(const GemmParams& p, long long batch_off, int row_base, int col0,
                                            int lane) {
  ChunkAt c;
  const int col = col0 + (lane & 3) * 4, row = row_base + (lane >> 2);
  c.off0 = batch_off + (long long)row * p.ldc + col;
  c.ok = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) c.ok |= (row + 8 * i < p.M && col < p.N ? 1u : 0u) << i;
  return c;
}

// One epilogue warp's chunks of a tile: 16 columns from `first` on, every `step`.  The accumulator (a
// row per TMEM lane) is waited for only after the first fused operands have been requested.
template <int MODE>
__device__ __forceinline__ bool drain_chunks(const CtaCtx& cx, const GemmParams& p, const CUtensorMap* tmC,
                                             const CUtensorMap* tmP, const TileCoord& tc, int warp, int lane,
                                             int acc, uint32_t acc_phase, uint32_t wait_code) {
  const int q = warp & 3;  // TMEM lane quarter this warp may read
  const int first = 16 * ((warp - 2) >> 2), step = 64, cols = p.bn, col0 = tc.n0;
  const uint32_t t_row = cx.tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(acc * ACC_COLS);
  uint8_t* stage = cx.epi_stage + (warp - 2) * EPI_STAGE_BYTES;
  const long long batch_off = (long long)tc.z0 * p.sC0 + (long long)tc.z1 * p.sC1;
  const int row_base = tc.m0 + q * 32;
  const bool tma_out = (MODE & E_NO_TMA) == 0 && p.tma_store != 0;
  float4 extra[4];
  const long long row8 = 8 * p.ldc;
  constexpr bool FETCH = (MODE & (E_DACT | E_RES)) != 0 && (MODE & E_GENERIC) == 0;
  if (FETCH) {
    const ChunkAt at = chunk_at(p, batch_off, row_base, col0 + first, lane);
    epilogue_fetch<MODE>(p, extra, at.off0, row8, at.ok);
  }
  if (!mbar_wait_warp(cx.tfull0 + 8 * acc, acc_phase, cx.abort_flag, p.err, wait_code + acc)) return false;
  tcgen05_fence_after();
  if ((MODE & E_NO_TMA) == 0 && tma_out) {
    if (row_base >= p.M) return true;
    const int end = min(cols, p.N - col0);           // chunks that start inside the matrix
    int c0 = first;
    if constexpr ((MODE & (E_F16 | E_BF16)) != 0 && (MODE & E_PRE) == 0) {
      for (; c0 + step < end; c0 += 2 * step) {
        uint32_t r[2][16];
        tmem_ld16(t_row + c0, r[0]);
        tmem_ld16(t_row + c0 + step, r[1]);
        tmem_wait_ld();
        epilogue_chunks_tma<MODE, 2>(p, tmC, tmP, r, stage, lane, col0 + c0, col0 + c0 + step, row_base,
                                     tc.z0, tc.z1);
      }
    }
    for (; c0 < end; c0 += step) {
      uint32_t r[1][16];
      tmem_ld16(t_row + c0, r[0]);
      tmem_wait_ld();
      epilogue_chunks_tma<MODE, 1>(p, tmC, tmP, r, stage, lane, col0 + c0, 0, row_base, tc.z0, tc.z1);
    }
    return true;
  }
  for (int c0 = first; c0 < cols; c0 += step) {
    if (col0 + c0 >= p.N) break;  // uniform across the warp
    uint32_t r[16];
    tmem_ld16(t_row + c0, r);
    tmem_wait_ld();
    // TMEM gives each lane one row; the chunk is transposed through shared memory so that global
    // loads and stores are row-contiguous (4 lanes x 16 B per row).  Rows are 64 B apart with the
    // 16-byte chunk index XOR-ed by (row >> 1) & 3: conflict-free both for the row-per-lane writes
    // and the row-contiguous reads.
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<uint4*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) =
          make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
    __syncwarp();
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = 8 * i + (lane >> 2);
      v[i] = *reinterpret_cast<const float4*>(stage + rr * 64 + (((lane & 3) ^ ((rr >> 1) & 3)) << 4));
    }
    float4 ex[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ex[i] = extra[i];
    if (FETCH && c0 + step < cols) {
      const ChunkAt at = chunk_at(p, batch_off, row_base, col0 + c0 + step, lane);
      epilogue_fetch<MODE>(p, extra, at.off0, row8, at.ok);
    }
    const ChunkAt at = chunk_at(p, batch_off, row_base, col0 + c0, lane);
    const int col = col0 + c0 + (lane & 3) * 4;
    const unsigned lanes = __ballot_sync(0xffffffffu, col < p.N);
    if (col < p.N)
      epilogue_chunk<MODE>(p, v, ex, at.off0, row8, at.ok, col, (tc.m0 / BM) * 4 + q, lanes);
    __syncwarp();
  }
  return true;
}

// Epilogue warp: drain this warp's share of the accumulator of work unit t.
template <int MODE>
__device__ __forceinline__ bool epilogue_unit(const CtaCtx& cx, const GemmParams& p,
                                              const CUtensorMap* tmC, const CUtensorMap* tmP, int t,
                                              int warp, int lane, int& acc, uint32_t& acc_phase) {
  const TileCoord tc = tile_coord(p, t);
  {
    int kb0, nkb;
    kb_range(p, tc, kb0, nkb);
    if (nkb <= 0) return true;
  }
  if (!drain_chunks<MODE>(cx, p, tmC, tmP, tc, warp, lane, acc, acc_phase, 0x400u)) return false;
  tcgen05_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(cx.tempty0 + 8 * acc);
  acc ^= 1;
  if (acc == 0) acc_phase ^= 1u;
  return true;
}

// Barriers, TMEM and the role-independent constants of a CTA.
// (Issuing the first loads here, before tensor memory is allocated, measured 1 us SLOWER per launch:
// the tensor maps prefetched at the top of the kernel are not there yet.)
__device__ __forceinline__ void cta_setup(CtaCtx& cx, uint8_t* smem_raw, const RingShape& ring) {
  // 128B-swizzled tiles want 1024-byte alignment.
  cx.base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (cx.base - smem_u32(smem_raw));
  cx.stage_bytes = (uint32_t)ring.stage_bytes;
  cx.n_stages = ring.stages;
  // Epilogue staging (one swizzled 32x16 fp32 chunk per epilogue warp), then the barrier block.
  cx.epi_stage = gen_base + RING_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(gen_base + RING_BYTES + EPI_WARPS * EPI_STAGE_BYTES);
  const uint32_t bar_base = cx.base + RING_BYTES + EPI_WARPS * EPI_STAGE_BYTES;
  // full[s] at +8s, empty[s] at +64+8s, tmem_full[a] at +128+8a, tmem_empty[a] at +144+8a
  cx.full0 = bar_base;
  cx.empty0 = bar_base + 64;
  cx.tfull0 = bar_base + 128;
  cx.tempty0 = bar_base + 144;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 20);
  cx.abort_flag = reinterpret_cast<volatile uint32_t*>(bars + 21);
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    for (int s = 0; s < cx.n_stages; ++s) {
      mbar_init(cx.full0 + 8 * s, 1);
      mbar_init(cx.empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(cx.tfull0 + 8 * a, 1);
      mbar_init(cx.tempty0 + 8 * a, EPI_WARPS);
    }
    *cx.abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void*)tmem_slot)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  cx.tmem_base = *tmem_slot;
}

// Teardown: everyone meets, then the allocating warp frees TMEM.
__device__ __forceinline__ void cta_teardown(const CtaCtx& cx) {
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (*cx.abort_flag) {
    // Give copies that may still be in flight time to land before the CTA's
    // shared memory is released.
    long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  if ((threadIdx.x >> 5) == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(cx.tmem_base),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

// One GEMM: CTA b takes tiles b, b + gridDim.x, ...
template <int MODE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                    const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmP,
                    const GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  pdl_trigger();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
    if ((MODE & E_NO_TMA) == 0 && p.tma_store) {
      prefetch_tensormap(&tmC);
      if (MODE & E_PRE) prefetch_tensormap(&tmP);
    }
  }
  CtaCtx cx;
  cta_setup(cx, smem_raw, RingShape(false, p.bn, p.b_mn & OP_MN, p.stage_kb));
  pdl_wait();      // barriers, TMEM and tensor maps are ready; operands may still be in flight
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int total_tiles = p.tiles_m * p.tiles_n * p.nb0 * (p.split_k > 1 ? p.split_k : p.nb1);
  if (warp == 0) {
    if (lane == 0) {
      Ring at;
      for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
        const TileCoord tc = tile_coord(p, t);
        if (!produce<false>(cx, p, &tmA, &tmB, tc, tc.n0, 0, at)) break;
      }
    }
  } else if (warp == 1) {
    Ring at;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x)
      if (!mma_unit<false>(cx, p, t, at, acc, acc_phase)) break;
  } else {
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = blockIdx.x; t < total_tiles; t += gridDim.x)
      if (!epilogue_unit<MODE>(cx, p, &tmC, &tmP, t, warp, lane, acc, acc_phase)) break;
    if (lane == 0) bulk_wait_read_all();   // the staging area outlives its last tile store
  }
  cta_teardown(cx);
}

// ---- grouped launch ------------------------------------------------------------------------
//
// Many independent GEMMs of the same tile width in one persistent launch: the dW = X^T dY of
// every Linear of a model, which have few tiles each (18..72 against 148 SMs) but thousands
// together.  Their tiles form one list, CTA b takes list entries b, b + gridDim.x, ...; with
// equal K (the rows of the batch) all entries cost the same, so the SMs stay level without
// splitting K and without a reduction pass.  The table lives in device memory: tensor maps,
// kernel parameters and the index of each problem's first list entry.
struct __align__(128) GroupEntry {
  CUtensorMap tmA, tmB, tmC;
  GemmParams p;
  int first_unit;
};
constexpr int GROUP_BN_SHIFT = 28;   // tile width code above the unit count of a grouped launch
constexpr int GROUP_MAX = 256;   // problems per launch (their first_unit values sit in shared memory)

// problem that list entry u belongs to: the last one whose first_unit is <= u
__device__ __forceinline__ int group_find(const int* first, int n, int u) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (first[mid] <= u) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_group_kernel(const GroupEntry* __restrict__ table, int n_problems, int total_units, int bn) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int first[GROUP_MAX];
  pdl_trigger();
  // the table was written by the host long before this launch, not by the kernel before it
  for (int i = threadIdx.x; i < n_problems; i += blockDim.x) first[i] = table[i].first_unit;
  CtaCtx cx;
  cta_setup(cx, smem_raw, RingShape(false, bn, true, table->p.stage_kb));   // its __syncthreads also publishes first[]
  pdl_wait();
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  if (warp == 0) {
    if (lane == 0) {
      Ring at;
      for (int u = blockIdx.x; u < total_units; u += gridDim.x) {
        const int pi = group_find(first, n_problems, u);
        const GemmParams p = table[pi].p;
        const TileCoord tc = tile_coord(p, u - first[pi]);
        if (!produce<false>(cx, p, &table[pi].tmA, &table[pi].tmB, tc, tc.n0, 0, at)) break;
      }
    }
  } else if (warp == 1) {
    Ring at;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int u = blockIdx.x; u < total_units; u += gridDim.x) {
      const int pi = group_find(first, n_problems, u);
      const GemmParams p = table[pi].p;
      if (!mma_unit<false>(cx, p, u - first[pi], at, acc, acc_phase)) break;
    }
  } else {
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int u = blockIdx.x; u < total_units; u += gridDim.x) {
      const int pi = group_find(first, n_problems, u);
      const GemmParams p = table[pi].p;
      if (!epilogue_unit<0>(cx, p, &table[pi].tmC, nullptr, u - first[pi], warp, lane, acc, acc_phase))
        break;
    }
    if (lane == 0) bulk_wait_read_all();
  }
  cta_teardown(cx);
}

// ---- CTA pairs -----------------------------------------------------------------------------
//
// 256 x 256 tiles on a 2-CTA cluster: each CTA loads its 128 rows of A and its 128 of the
// tile's 256 columns of B, the even-ranked CTA issues tcgen05.mma.cta_group::2 for both, and
// each CTA's TMEM receives the accumulators of its own 128 rows.  Per k-block a CTA pulls
// 32 KB through L2 instead of 48 KB for the same 128 x 256 outputs, which is what bounds the
// single-CTA kernel on the K = 768 shapes.  Barriers: TMA of both CTAs counts bytes on the
// leader's full[s]; the leader's commits arrive on empty[s] / tmem_full[a] of both CTAs;
// the epilogue warps of both CTAs arrive on the leader's tmem_empty[a].
constexpr int PAIR_BN = 256;        // widest pair tile; 192 is the other width (N = 768 shapes)
// Barriers, TMEM and constants of one CTA of a pair; ends with a cluster-wide barrier so the
// peer's mbarriers exist before anything is signalled on them.
__device__ __forceinline__ void pair_setup(CtaCtx& cx, uint8_t* smem_raw, const RingShape& ring) {
  const int warp = threadIdx.x >> 5;
  cx.base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen_base = smem_raw + (cx.base - smem_u32(smem_raw));
  cx.stage_bytes = (uint32_t)ring.stage_bytes;
  cx.n_stages = ring.stages;
  cx.epi_stage = gen_base + RING_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(gen_base + RING_BYTES + EPI_WARPS * EPI_STAGE_BYTES);
  const uint32_t bar_base = cx.base + RING_BYTES + EPI_WARPS * EPI_STAGE_BYTES;
  cx.full0 = bar_base;
  cx.empty0 = bar_base + 64;
  cx.tfull0 = bar_base + 128;
  cx.tempty0 = bar_base + 144;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + 20);
  cx.abort_flag = reinterpret_cast<volatile uint32_t*>(bars + 21);
  if (threadIdx.x == 0) {
    for (int s = 0; s < cx.n_stages; ++s) {
      mbar_init(cx.full0 + 8 * s, 1);     // the leader's own arrive.expect_tx
      mbar_init(cx.empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(cx.tfull0 + 8 * a, 1);
      mbar_init(cx.tempty0 + 8 * a, 2 * EPI_WARPS);   // the epilogue warps of both CTAs
    }
    *cx.abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    // each CTA takes the whole of its own TMEM, so accumulator addresses agree in the pair
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32((const void*)tmem_slot)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();        // the peer's barriers exist before anything is signalled on them
  tcgen05_fence_after();
  cx.tmem_base = *tmem_slot;

}

// Neither CTA may leave while the other can still read its shared memory or signal its
// barriers.
__device__ __forceinline__ void pair_teardown(const CtaCtx& cx) {
  const int warp = threadIdx.x >> 5;
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (*cx.abort_flag) {
    long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  if (warp == 1) {
    tcgen05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(cx.tmem_base),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

// Tile t as CTA `rank` of the pair sees it: its 128 rows of A, and its half of the columns of B.
__device__ __forceinline__ TileCoord pair_coord(const GemmParams& p, int t, uint32_t rank) {
  return tile_coord(p, t, 2 * BM, (int)rank * BM);
}

// Epilogue warp of one CTA of the pair: its 128 rows of the 256 x 256 tile.
template <int MODE>
__device__ __forceinline__ bool pair_epilogue_unit(const CtaCtx& cx, const GemmParams& p,
                                                   const CUtensorMap* tmC, const CUtensorMap* tmP, int t,
                                                   uint32_t rank, int warp, int lane, int& acc,
                                                   uint32_t& acc_phase) {
  const TileCoord tc = pair_coord(p, t, rank);
  {
    int kb0, nkb;
    kb_range(p, tc, kb0, nkb);
    if (nkb <= 0) return true;
  }
  if (!drain_chunks<MODE>(cx, p, tmC, tmP, tc, warp, lane, acc, acc_phase, 0x800u)) return false;
  tcgen05_fence_before();
  __syncwarp();
  if (lane == 0) {
    if (rank == 0) mbar_arrive(cx.tempty0 + 8 * acc);
    else mbar_arrive_cluster(mapa_shared(cx.tempty0 + 8 * acc, 0));
  }
  acc ^= 1;
  if (acc == 0) acc_phase ^= 1u;
  return true;
}

template <int MODE>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_cta_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                     const __grid_constant__ CUtensorMap tmC, const __grid_constant__ CUtensorMap tmP,
                     const GemmParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  pdl_trigger();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmA);
    prefetch_tensormap(&tmB);
    if ((MODE & E_NO_TMA) == 0 && p.tma_store) {
      prefetch_tensormap(&tmC);
      if (MODE & E_PRE) prefetch_tensormap(&tmP);
    }
  }
  CtaCtx cx;
  pair_setup(cx, smem_raw, RingShape(true, p.bn, p.b_mn & OP_MN, p.stage_kb));
  pdl_wait();
  const int n_pairs = (int)gridDim.x >> 1, pair = (int)blockIdx.x >> 1;
  const int total_tiles = p.tiles_m * p.tiles_n * p.nb0 * (p.split_k > 1 ? p.split_k : p.nb1);
  if (warp == 0) {
    Ring at;
    for (int t = pair; t < total_tiles; t += n_pairs) {
      const TileCoord tc = pair_coord(p, t, rank);
      if (!produce<true>(cx, p, &tmA, &tmB, tc, tc.n0 + (int)rank * (p.bn / 2), rank, at)) break;
    }
  } else if (warp == 1) {
    if (rank == 0) {
      Ring at;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int t = pair; t < total_tiles; t += n_pairs)
        if (!mma_unit<true>(cx, p, t, at, acc, acc_phase)) break;
    }
  } else {
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int t = pair; t < total_tiles; t += n_pairs)
      if (!pair_epilogue_unit<MODE>(cx, p, &tmC, &tmP, t, rank, warp, lane, acc, acc_phase)) break;
    if (lane == 0) bulk_wait_read_all();
  }
  pair_teardown(cx);
}

// The grouped launch on CTA pairs: list entries are 256 x 256 tiles.
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_group_pair_kernel(const GroupEntry* __restrict__ table, int n_problems, int total_units) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  __shared__ int first[GROUP_MAX];
  pdl_trigger();
  for (int i = threadIdx.x; i < n_problems; i += blockDim.x) first[i] = table[i].first_unit;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  CtaCtx cx;
  pair_setup(cx, smem_raw, RingShape(true, PAIR_BN, true, 1));   // publishes first[]
  pdl_wait();
  const int n_pairs = (int)gridDim.x >> 1, pair = (int)blockIdx.x >> 1;
  if (warp == 0) {
    Ring at;
    for (int u = pair; u < total_units; u += n_pairs) {
      const int pi = group_find(first, n_problems, u);
      const GemmParams p = table[pi].p;
      const TileCoord tc = pair_coord(p, u - first[pi], rank);
      if (!produce<true>(cx, p, &table[pi].tmA, &table[pi].tmB, tc, tc.n0 + (int)rank * (p.bn / 2), rank, at)) break;
    }
  } else if (warp == 1) {
    if (rank == 0) {
      Ring at;
      int acc = 0;
      uint32_t acc_phase = 0;
      for (int u = pair; u < total_units; u += n_pairs) {
        const int pi = group_find(first, n_problems, u);
        const GemmParams p = table[pi].p;
        if (!mma_unit<true>(cx, p, u - first[pi], at, acc, acc_phase)) break;
      }
    }
  } else {
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int u = pair; u < total_units; u += n_pairs) {
      const int pi = group_find(first, n_problems, u);
      const GemmParams p = table[pi].p;
      if (!pair_epilogue_unit<0>(cx, p, &table[pi].tmC, nullptr, u - first[pi], rank, warp, lane, acc,
                                 acc_phase))
        break;
    }
    if (lane == 0) bulk_wait_read_all();
  }
  pair_teardown(cx);
}

// Adds the K slices of a split GEMM in slice order and writes C (fp32, row pitch ldc).
__global__ void k_splitk_reduce(const float4* __restrict__ ws, float* __restrict__ C, int M, int N4,
                                long long ldc, int splits) {
  pdl_trigger();
  pdl_wait();
  const long long per = (long long)M * N4;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < per;
       i += (long long)gridDim.x * blockDim.x) {
    float4 a = ws[i];
    for (int s = 1; s < splits; ++s) {
      const float4 b = ws[i + s * per];
      a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    }
    const long long r = i / N4, c = i - r * N4;
    *reinterpret_cast<float4*>(C + r * ldc + c * 4) = a;
  }
}

typedef void (*GemmKernel)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                           const GemmParams);
struct Specialised {
  int mode;
  GemmKernel fn;
};
#define VKG_SPEC(m) {(m), gemm_tcgen05_kernel<(m)>}
// The epilogues the training step uses; anything else runs the generic kernel.
const Specialised kSpecialised[] = {
    VKG_SPEC(0),                                   // fp32 out: dW, dX into layernorm, scores
    VKG_SPEC(E_F16),                               // fp16 out: attention products, dO
    VKG_SPEC(E_BIAS),                              // fp32 out + bias: logits of an untied head
    VKG_SPEC(E_BIAS | E_F16),                      // qkv projection
    VKG_SPEC(E_BIAS | E_RES),                      // proj / fc2 forward: + bias + residual
    VKG_SPEC(E_BIAS | E_PRE | E_ACT | E_F16),      // fc1 forward: bias, keep z, GELU, narrow
    VKG_SPEC(E_BIAS | E_ACT | E_F16),              // the same without a backward to keep z for
    VKG_SPEC(E_DACT | E_F16),                      // fc2 dX: * GELU'(z), narrow
    VKG_SPEC(E_DACT | E_F16 | E_COLSUM),           // the same + column sums = fc1's bias gradient
    VKG_SPEC(E_GENERIC),                           // last: whatever is not above
};
const int kNumSpecialised = sizeof(kSpecialised) / sizeof(kSpecialised[0]);
#define VKG_SPEC_CP(m) {(m), gemm_cta_pair_kernel<(m)>}
// The same epilogues on 256 x 256 tiles computed by CTA pairs.
const Specialised kCtaPair[] = {
    VKG_SPEC_CP(0),
    VKG_SPEC_CP(E_F16),
    VKG_SPEC_CP(E_BIAS),
    VKG_SPEC_CP(E_BIAS | E_F16),
    VKG_SPEC_CP(E_BIAS | E_RES),
    VKG_SPEC_CP(E_BIAS | E_PRE | E_ACT | E_F16),
    VKG_SPEC_CP(E_BIAS | E_ACT | E_F16),
    VKG_SPEC_CP(E_DACT | E_F16),
    VKG_SPEC_CP(E_DACT | E_F16 | E_COLSUM),
    VKG_SPEC_CP(E_GENERIC),
};
const int kNumCtaPair = sizeof(kCtaPair) / sizeof(kCtaPair[0]);
GemmKernel pick(const Specialised* t, int n, int mode) {
  int i = 0;
  while (i + 1 < n && t[i].mode != mode) ++i;
  return t[i].fn;
}
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 5-D map over a 16-bit matrix with two batch strides: {inner, rows, 1, nb0, nb1}, or wide (Feed)
// {64, rows, inner / 64, nb0, nb1}, with boxes of 64 x box_rows x pieces.
int make_map(vkg_device* dev, CUtensorMap* map, const void* ptr, int dtype, int64_t inner,
             int64_t rows, int64_t ld, int nb0, int64_t s0, int nb1, int64_t s1, bool wide, int box_rows,
             int pieces, const char* what) {
  cuuint64_t dims[5] = {(cuuint64_t)(wide ? 64 : inner), (cuuint64_t)rows, (cuuint64_t)(wide ? inner / 64 : 1),
                        (cuuint64_t)nb0, (cuuint64_t)nb1};
  int64_t pitch = ld * 2;
  int64_t st0 = nb0 > 1 ? s0 * 2 : pitch * rows;
  int64_t st1 = nb1 > 1 ? s1 * 2 : (nb0 > 1 ? st0 * nb0 : pitch * rows);
  cuuint64_t strides[4] = {(cuuint64_t)pitch, (cuuint64_t)(wide ? 128 : pitch * rows), (cuuint64_t)st0,
                           (cuuint64_t)st1};
  cuuint32_t box[5] = {64, (cuuint32_t)box_rows, (cuuint32_t)pieces, 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  if (((uintptr_t)ptr & 15) || (pitch & 15) || (st0 & 15) || (st1 & 15)) {
    vkg_set_error("gemm operand %s: base address and strides must be multiples of 16 bytes "
                  "(ptr %p, ld %lld, batch strides %lld/%lld elements)",
                  what, ptr, (long long)ld, (long long)s0, (long long)s1);
    return 1;
  }
  CUresult r = ((EncodeTiledFn)dev->encode_tiled)(
      map, dtype == VKG_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5,
      const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    vkg_set_error("cuTensorMapEncodeTiled failed for operand %s with code %d", what, (int)r);
    return 1;
  }
  return 0;
}

// 4-D map {N, M, nb0, nb1} over the output (fp32 or 16-bit) for the epilogue's tile stores:
// boxes of 16 columns x 32 rows in the 64-byte (fp32) or 32-byte (16-bit) swizzle the staging
// area is written in.  *ok = false (and no error) when the layout cannot be described: the
// epilogue then stores per lane.
int make_out_map(vkg_device* dev, CUtensorMap* map, const void* ptr, int dtype, int64_t n_cols,
                 int64_t n_rows, int64_t ld, int nb0, int64_t s0, int nb1, int64_t s1, bool* ok) {
  *ok = false;
  const int64_t es = dtype == VKG_F32 ? 4 : 2;
  const int64_t pitch = ld * es;
  const int64_t st0 = nb0 > 1 ? s0 * es : pitch * n_rows;
  const int64_t st1 = nb1 > 1 ? s1 * es : (nb0 > 1 ? st0 * nb0 : pitch * n_rows);
  if (((uintptr_t)ptr & 15) || (pitch & 15) || (st0 & 15) || (st1 & 15) || st0 <= 0 || st1 <= 0 ||
      pitch >= (1ll << 40) || st0 >= (1ll << 40) || st1 >= (1ll << 40))
    return 0;
  cuuint64_t dims[4] = {(cuuint64_t)n_cols, (cuuint64_t)n_rows, (cuuint64_t)nb0, (cuuint64_t)nb1};
  cuuint64_t strides[3] = {(cuuint64_t)pitch, (cuuint64_t)st0, (cuuint64_t)st1};
  cuuint32_t box[4] = {16, 32, 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  const CUtensorMapDataType dt = dtype == VKG_F32    ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                 : dtype == VKG_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16
                                                     : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  CUresult r = ((EncodeTiledFn)dev->encode_tiled)(
      map, dt, 4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
      es == 4 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    vkg_set_error("cuTensorMapEncodeTiled failed for the output map with code %d", (int)r);
    return 1;
  }
  *ok = true;
  return 0;
}

// ---- which tiles ---------------------------------------------------------------------------
//
// A launch is planned with a time model over its candidates: 128-row tiles of one CTA and 256-row
// tiles of a CTA pair, 64 to 256 columns wide.  How many slices K is cut into is not the model's to
// choose (k_slices): it is part of the result.  Its constants were fitted to 208 shapes (M to 50272,
// N and K alike, aligned and ragged, the three transpositions, every epilogue of a training step;
// launches in a graph on B200, operands warm) when a k-block of a narrow tile still took a load and a wait
// of its own; since then they are too high there, by a quarter, but the order they give stands: over
// 380 drawn shapes the choice takes 0.4 % longer than the best candidate on average, more than 5 % for nine,
// 1.35 times as long at worst.
// Constants fitted anew, 10 % off the times instead of 18 %, chose no better (0.3 % on shapes held out; a block
// run through the op dictionaries 261 us against 259).
//
// Per k-block (64 of K), microseconds by tile width 64 / 128 / 192 / 256.  A CTA pulls its operands
// through an L2 port of 64 bytes a cycle; K-major operands go a little faster than MN-major ones.
struct KBlockCost {
  double single[4], pair[2];     // pair: 192, 256
};
constexpr KBlockCost KB_NN = {{0.225, 0.270, 0.305, 0.375}, {0.315, 0.375}};
constexpr KBlockCost KB_NT = {{0.185, 0.235, 0.270, 0.345}, {0.300, 0.370}};
constexpr KBlockCost KB_TN = {{0.245, 0.300, 0.335, 0.400}, {0.330, 0.375}};
constexpr double PL_LAUNCH = 3.43;     // launch, set-up, first load, drain
constexpr double PL_EPI = 0.69, PL_EPI_COL = 0.00658;   // epilogue of a tile, per column at fp32 out
constexpr double PL_PAIR = 1.29;       // a pair's barriers and its later start
// A launch that overlaps its predecessor, whatever its waves.  In this model's time: 9 to 10 us measured.
constexpr double PL_SHORT_US = 12.0;
constexpr double PL_IDLE = 0.81;       // k-block cost with one CTA busy, of that with all
constexpr double PL_WAVE = 0.95;       // per further wave
constexpr double PL_OVERLAP = 1.42;    // epilogue beside a main loop, of the epilogue alone
constexpr double PL_RAGGED[2] = {0.387, 0.138};   // operand rows off the 128-byte lines: single, pair
constexpr double PL_HOT[2] = {0.293, 0.064};      // the clock under sustained load: single, pair
constexpr double PL_HOT_FLOPS = 3.5e10;

struct Tiles {
  bool pair;
  int bn, split;
  double us;
};

double tiles_us(const vkg_gemm_args* a, bool pair, int bn, int split, int batch, int slots) {
  const double M = a->M, N = a->N, K = a->K;
  const int kbs = ((a->K + BK - 1) / BK + split - 1) / split;
  const int bm = pair ? 2 * BM : BM;
  const long long tiles = (long long)((a->M + bm - 1) / bm) * ((a->N + bn - 1) / bn) * batch * split;
  const KBlockCost& kb = a->trans_a ? KB_TN : a->trans_b ? KB_NT : KB_NN;
  double tk = pair ? kb.pair[bn / 64 - 3] : kb.single[bn / 64 - 1];
  const double busy = tiles < slots ? (double)tiles / slots : 1.0;
  tk *= PL_IDLE + (1.0 - PL_IDLE) * busy;
  // operand bytes of a k-block whose rows do not start on 128-byte lines
  const double rows_a = BM, rows_b = pair ? bn / 2 : bn;
  const double ragged = ((a->lda % 64 ? rows_a : 0) + (a->ldb % 64 ? rows_b : 0)) / (rows_a + rows_b);
  const double flops = 2.0 * M * N * K * batch;
  const double hot = flops < PL_HOT_FLOPS ? flops / PL_HOT_FLOPS : 1.0;
  tk *= (1.0 + PL_RAGGED[pair] * ragged) * (1.0 + PL_HOT[pair] * hot);
  // bytes an output element costs the epilogue, written and read; the column sums count two
  const int out = split > 1 ? 4
                            : (a->c_dtype == VKG_F32 ? 4 : 2) + (a->pre ? 4 : 0) + (a->dact_z ? 4 : 0) +
                                  (a->residual ? 4 : 0) + (a->C2 ? 2 : 0) + (a->colsum ? 2 : 0);
  const double epi = PL_EPI + (pair ? PL_PAIR : 0.0) + PL_EPI_COL * bn * (0.5 + 0.125 * out);
  const double main_loop = kbs * tk;
  const long long waves = (tiles + slots - 1) / slots;
  return PL_LAUNCH + main_loop + epi +
         (waves - 1) * (main_loop + PL_WAVE > epi * PL_OVERLAP ? main_loop + PL_WAVE : epi * PL_OVERLAP);
}

// single / pair: whether such tiles may be used; force_bn: 0 = free; split: slices of K.
Tiles choose_tiles(vkg_device* dev, const vkg_gemm_args* a, bool single, bool pair, int force_bn, int split) {
  const int batch = (a->nb0 > 0 ? a->nb0 : 1) * (a->nb1 > 0 ? a->nb1 : 1);
  const int n_round = ((a->N + 63) / 64) * 64;
  const int ctas = a->max_ctas > 0 ? a->max_ctas : vkg_persistent_ctas(dev);
  Tiles best = {false, 64, split, -1.0};
  for (int kind = 0; kind < 2; ++kind) {
    if (kind ? !pair : !single) continue;
    for (int bn = kind ? 192 : 64; bn <= 256; bn += 64) {
      if (force_bn ? bn != force_bn : bn > n_round && bn != 64) continue;
      if (kind && !force_bn && a->cta_pair <= 0 && bn == 192 && !dev->pair192) continue;
      const int slots = kind ? ctas / 2 : ctas;
      if (slots < 1) continue;
      const double us = tiles_us(a, kind != 0, bn, split, batch, slots);
      if (kind && bn == 256 && split == 1 && a->cta_pair <= 0 && dev->pair_min_waves_x10 > 0) {
        const long long tiles = (long long)((a->M + 2 * BM - 1) / (2 * BM)) * ((a->N + bn - 1) / bn) * batch;
        if (10 * tiles < (long long)dev->pair_min_waves_x10 * slots) continue;
      }
      if (best.us < 0 || us < best.us) best = {kind != 0, bn, split, us};
    }
  }
  return best;
}

// Whether an output is one that slices of K can be added up into: fp32, not batched, nothing in the
// epilogue.
bool plain_output(const vkg_gemm_args* a) {
  const int batch = (a->nb0 > 0 ? a->nb0 : 1) * (a->nb1 > 0 ? a->nb1 : 1);
  return !a->bias && !a->pre && !a->act && !a->dact_z && !a->residual && !a->C2 && !a->colsum &&
         a->c_dtype == VKG_F32 && (a->alpha == 0.0f || a->alpha == 1.0f) && batch == 1 && a->causal == 0 &&
         a->N % 4 == 0 && a->ldc % 4 == 0 && ((uintptr_t)a->C & 15) == 0;
}

// Whether K may be cut into slices that a second launch adds up.
bool may_split(const vkg_gemm_args* a) {
  return plain_output(a) && a->workspace && ((uintptr_t)a->workspace & 15) == 0;
}

// Slices of K where the caller leaves them to the library: a rule of M, N, K and the tiles the caller
// insists on.  Nothing else may enter it -- not the time model above, not how many SMs a launch is
// held to, not how large a workspace happens to be: slices change the order of a sum, by 1e-6 of the
// result, and a training step whose fp16 gradients are subnormals, for want of a loss scale, makes
// 2e-3 of that in its second step (512-wide model, 1800 rows: the head's dW).  The rule: few
// 256-column pair tiles, or few single ones, are cut while that shortens the waves of a full B200 by
// more than the reduction costs, by the k-block and epilogue times of an early version of the kernel.
constexpr int SLICE_SMS = 148, SLICE_MAX = 16;
int k_slices(const vkg_gemm_args* a) {
  const int num_kb = (a->K + BK - 1) / BK, n_round = ((a->N + 63) / 64) * 64;
  const int64_t out_bytes = (int64_t)a->M * a->N * 4;
  const auto slices = [&](int bm, int slots, int only_bn) {
    double best = -1.0;
    int got = 1;
    for (int bn = 256; bn >= 64; bn -= 64) {
      if (only_bn ? bn != only_bn : bn > n_round && bn != 64) continue;
      const long long tiles = (long long)((a->M + bm - 1) / bm) * ((a->N + bn - 1) / bn);
      const double t_kb = bn == 256 ? 0.41 : bn == 192 ? 0.36 : 0.33;
      for (int sp = 1; sp <= SLICE_MAX; ++sp) {
        if (sp > 1 && num_kb / sp < 4) break;
        const long long waves = (tiles * sp + slots - 1) / slots;
        double t = waves * ((num_kb + sp - 1) / sp * t_kb + 4.4 * bn / 256.0);
        if (sp > 1) t += (double)(sp + 1) * out_bytes / 4.0e6 + 4.0;
        if (best < 0 || t < best) {
          best = t;
          got = sp;
        }
      }
    }
    return got;
  };
  const bool any = a->split_k < 0;      // -1: as if the tiles were the library's to choose
  const int tile_n = any ? 0 : a->tile_n, pair = any ? 0 : a->cta_pair;
  if (pair >= 0 && a->M > BM && a->N >= PAIR_BN / 2 && (tile_n == 0 || tile_n == 192 || tile_n == PAIR_BN) &&
      (any || a->max_ctas == 0)) {
    const long long rows = (a->M + 2 * BM - 1) / (2 * BM);
    const int slots = SLICE_SMS / 2;
    if (pair > 0 || slices(2 * BM, slots, PAIR_BN) > 1 || 10 * rows * ((a->N + 255) / 256) >= 60ll * slots)
      return slices(2 * BM, slots, tile_n == 192 ? 192 : PAIR_BN);
    if (tile_n == 0 && a->N % 192 == 0 && a->N <= 4 * 192 && a->K >= 1536 && rows * (a->N / 192) >= slots)
      return slices(2 * BM, slots, 192);
  }
  return slices(BM, SLICE_SMS, tile_n);
}

// One width for all problems of a grouped launch, from the same costs: waves of all their tiles
// together.  256-wide pair tiles of six 384-wide layers' dW leave half of their third wave empty and
// pad 384 columns to 512: 65 us, with the width chosen here 55.
Tiles choose_group_tiles(vkg_device* dev, const vkg_gemm_args* args, int n, bool pair_ok) {
  Tiles best = {false, 256, 1, -1.0};
  for (int kind = 0; kind < (pair_ok ? 2 : 1); ++kind) {
    for (int bn = kind ? 256 : 64; bn <= 256; bn += 64) {
      const int bm = kind ? 2 * BM : BM, slots = vkg_persistent_ctas(dev) / (kind ? 2 : 1);
      long long units = 0;
      double work = 0.0, longest = 0.0, flops = 0.0;
      for (int i = 0; i < n; ++i) flops += 2.0 * args[i].M * args[i].N * args[i].K;
      const double hot = 1.0 + PL_HOT[kind] * (flops < PL_HOT_FLOPS ? flops / PL_HOT_FLOPS : 1.0);
      for (int i = 0; i < n; ++i) {
        const vkg_gemm_args* a = &args[i];
        const KBlockCost& kb = a->trans_a ? KB_TN : a->trans_b ? KB_NT : KB_NN;
        const long long t = (long long)((a->M + bm - 1) / bm) * ((a->N + bn - 1) / bn);
        const double tk = kind ? kb.pair[bn / 64 - 3] : kb.single[bn / 64 - 1];
        const double one = (double)((a->K + BK - 1) / BK) * tk * hot + PL_WAVE;
        units += t;
        work += t * one;
        longest = one > longest ? one : longest;
      }
      if (slots < 1 || units < 1) continue;
      const long long waves = (units + slots - 1) / slots;
      const double wave = work / units > longest * 0.99 ? longest : work / units;
      const double us = PL_LAUNCH + PL_EPI + (kind ? PL_PAIR : 0.0) + PL_EPI_COL * bn + waves * wave;
      if (best.us < 0 || us < best.us) best = {kind != 0, bn, 1, us};
    }
  }
  return best;
}

// One GEMM made ready to launch: kernel parameters, operand maps, epilogue mask.
struct Problem {
  GemmParams p;
  CUtensorMap tmA, tmB, tmC, tmP;
  int mode;
  bool vec;
  long long total_tiles;
};

// The arguments' own conditions, before anything is planned from them.
int check_args(const vkg_gemm_args* a) {
  VKG_REQUIRE(a, "null gemm args");
  VKG_REQUIRE(a->M > 0 && a->N > 0 && a->K > 0, "gemm: M, N, K must be positive (%d, %d, %d)",
              a->M, a->N, a->K);
  VKG_REQUIRE(a->N % 8 == 0, "gemm: N must be a multiple of 8 (got %d)", a->N);
  VKG_REQUIRE(a->in_dtype == VKG_F16 || a->in_dtype == VKG_BF16,
              "gemm: inputs must be f16 or bf16");
  VKG_REQUIRE(a->c_dtype == VKG_F32 || a->c_dtype == VKG_F16 || a->c_dtype == VKG_BF16,
              "gemm: unknown output dtype %d", a->c_dtype);
  VKG_REQUIRE(a->A && a->B && a->C, "gemm: null operand");
  VKG_REQUIRE(a->causal >= 0 && a->causal <= 3, "gemm: causal mode %d unknown", a->causal);
  VKG_REQUIRE(a->ldc >= a->N, "gemm: ldc %lld < N %d", (long long)a->ldc, a->N);

  VKG_REQUIRE(a->tile_n == 0 || a->tile_n == 64 || a->tile_n == 128 || a->tile_n == 192 ||
                  a->tile_n == 256, "gemm: tile_n %d not in {64,128,192,256}", a->tile_n);
  VKG_REQUIRE(a->split_k <= 1 || may_split(a),
              "gemm: split_k needs an unbatched GEMM with a plain fp32 output, a 16-byte aligned "
              "workspace, and N, ldc multiples of 4");
  return 0;
}

// Two k-blocks to a stage where that leaves three stages (the 192-wide pair tile does too).
int most_stage_kb(bool pair, int bn) {
  return pair ? (bn == PAIR_BN ? 1 : 2) : RING_BYTES / (2 * (A_STAGE_BYTES + bn * 128)) >= 3 ? 2 : 1;
}

// Whether a launch takes them: kbs k-blocks to a work unit, operands wide (Feed) or in pieces.  Two save a wait
// and, of all but K-major operands in pieces, loads; but the first products wait for both, 0.1 us later.
// Against a start with one k-block to a stage, 88 drawn shapes in three transpositions:
//   - one k-block to a unit: the second is loaded for nothing (2822 x 64 x 400 NN 4.35 us, with two 4.70);
//   - all in pieces, both K-major: two save no load (1545 x 80 x 264 NT 3.90, with two 4.02);
//   - all in pieces, single tiles: of the loads saved a tile of 64 columns sees little (837 x 280 x 264 NN 4.92,
//     with two 5.01; 264 x 1544 x 80 TN 6.03, 6.26), wider MN-major ones do, and pairs (1760 x 3304 x 1904 TN
//     24.2, with two 19.9);
//   - both only up to ten k-blocks to a unit: calls one at a time lose beyond (1058 x 816 x 848 NT, thirteen:
//     7.78, with two 7.62; 600 x 1992 x 3336 NT 18.0, 17.4), though launches in a row gain up to 2 % there;
//   - one in pieces: two pay from five k-blocks on (915 x 736 x 128 NN 5.67, with two 5.34), where a K-major one
//     is, else from four (248 x 168 x 1344 TN, three: 4.17, with two 4.42).
// The kernel of before those loads took 4.35, 3.88, 4.91, 5.98 and 24.2 us, 7.78, 17.6, 6.1 and 4.18.
int stage_kb_for(const vkg_gemm_args* a, bool pair, int bn, int kbs, bool a_wide, bool b_wide) {
  if (most_stage_kb(pair, bn) == 1 || kbs <= 1) return 1;
  if (a_wide && b_wide) return 2;
  const bool k_pieces = (!a->trans_a && !a_wide) || (a->trans_b && !b_wide);
  if (a_wide || b_wide) return kbs <= (k_pieces ? 4 : 3) ? 1 : 2;
  const bool saves_little = (!a->trans_a && a->trans_b) || (!pair && (k_pieces || bn == 64));
  return saves_little && kbs <= 10 ? 1 : 2;
}

// use_pair: 256 x bn tiles for gemm_cta_pair_kernel (the caller has checked the shape).  grouped: the ring is
// shared with other problems.
int build_problem(vkg_device* dev, const vkg_gemm_args* a, Problem* out, bool use_pair, int bn, int want_split,
                  bool grouped = false) {
  if (check_args(a)) return 1;
  const int nb0 = a->nb0 > 0 ? a->nb0 : 1, nb1 = a->nb1 > 0 ? a->nb1 : 1;
  const int batch = nb0 * nb1;
  const int bm = use_pair ? 2 * BM : BM;

  GemmParams& p = out->p;
  memset(&p, 0, sizeof(p));
  p.M = a->M; p.N = a->N; p.K = a->K;
  p.nb0 = nb0; p.nb1 = nb1;
  p.tiles_m = (a->M + bm - 1) / bm;
  p.tiles_n = (a->N + bn - 1) / bn;
  p.bn = bn;
  p.num_kb = (a->K + BK - 1) / BK;
  const int rows_b = use_pair ? bn / 2 : bn, b_groups = (rows_b + 63) / 64;
  const bool a_wide = (a->trans_a ? a->M : a->K) % 64 == 0;
  const bool b_wide = (a->trans_b ? a->K : a->N) % 64 == 0 && (a->trans_b || rows_b % 64 == 0);
  const int kbs = want_split > 1 ? (p.num_kb + want_split - 1) / want_split : p.num_kb;
  p.stage_kb = grouped ? most_stage_kb(use_pair, bn) : stage_kb_for(a, use_pair, bn, kbs, a_wide, b_wide);
  p.a_mn = (a->trans_a ? OP_MN : 0) | (a_wide ? OP_WIDE : 0);
  p.b_mn = (a->trans_b ? 0 : OP_MN) | (b_wide ? OP_WIDE : 0);
  const uint32_t fmt = a->in_dtype == VKG_BF16 ? 1u : 0u;
  p.idesc = (1u << 4) | (fmt << 7) | (fmt << 10) | ((uint32_t)(p.a_mn & OP_MN) << 15) |
            ((uint32_t)(p.b_mn & OP_MN) << 16) | ((uint32_t)(bn >> 3) << 17) | ((uint32_t)(bm >> 4) << 24);
  p.c_dtype = a->c_dtype; p.act = a->act; p.dact = a->dact;
  p.ldc = a->ldc; p.sC0 = a->sC0; p.sC1 = a->sC1;
  p.C = a->C; p.C2 = a->C2; p.bias = a->bias; p.pre = a->pre;
  p.dact_z = a->dact_z; p.residual = a->residual;
  if (a->colsum) {
    VKG_REQUIRE(a->colsum_scratch && batch == 1 && a->causal == 0 && a->split_k <= 1,
                "gemm: colsum needs colsum_scratch, one matrix, causal == 0 and an unsplit K");
    p.colsum = a->colsum_scratch;
  }
  p.alpha = a->alpha == 0.0f ? 1.0f : a->alpha;
  p.err = dev->err_dev;
  p.split_k = 1;
  p.kb_per_split = p.num_kb;
  p.causal = a->causal;
  if (want_split > 1) {
    int splits = want_split < p.num_kb ? want_split : p.num_kb;
    p.kb_per_split = (p.num_kb + splits - 1) / splits;
    splits = (p.num_kb + p.kb_per_split - 1) / p.kb_per_split;   // no empty slice
    if (splits > 1) {
      VKG_REQUIRE(a->workspace_bytes >= (int64_t)splits * a->M * a->N * 4,
                  "gemm: split_k workspace too small (%lld bytes for %d slices of %d x %d)",
                  (long long)a->workspace_bytes, splits, a->M, a->N);
      p.split_k = splits;
      p.C = a->workspace;
      p.ldc = a->N;
      p.sC0 = 0;
      p.sC1 = (long long)a->M * a->N;
    }
  }
  // 16-byte vector accesses in the epilogue need every touched array aligned
  // for its element width at every (row, 8-column group).
  bool vec = (a->ldc % 4 == 0) && (a->sC0 % 4 == 0) && (a->sC1 % 4 == 0);
  const void* ptrs[6] = {a->C, a->C2, a->pre, a->dact_z, a->residual, a->bias};
  for (int i = 0; i < 6; ++i)
    if (ptrs[i] && ((uintptr_t)ptrs[i] & 15)) vec = false;
  p.vec_ok = vec ? 1 : 0;

  CUtensorMap& tmA = out->tmA;
  CUtensorMap& tmB = out->tmB;
  if (!a->trans_a) {
    VKG_REQUIRE(a->lda >= a->K, "gemm: lda %lld < K %d", (long long)a->lda, a->K);
    if (make_map(dev, &tmA, a->A, a->in_dtype, a->K, a->M, a->lda, nb0, a->sA0, nb1, a->sA1, a_wide, BM,
                 a_wide ? p.stage_kb : 1, "A"))
      return 1;
  } else {
    VKG_REQUIRE(a->lda >= a->M, "gemm: lda %lld < M %d (A stored K x M)", (long long)a->lda, a->M);
    if (make_map(dev, &tmA, a->A, a->in_dtype, a->M, a->K, a->lda, nb0, a->sA0, nb1, a->sA1, a_wide,
                 p.stage_kb * BK, a_wide ? BM / 64 : 1, "A^T"))
      return 1;
  }
  if (a->trans_b) {
    VKG_REQUIRE(a->ldb >= a->K, "gemm: ldb %lld < K %d (B stored N x K)", (long long)a->ldb, a->K);
    if (make_map(dev, &tmB, a->B, a->in_dtype, a->K, a->N, a->ldb, nb0, a->sB0, nb1, a->sB1, b_wide,
                 rows_b, b_wide ? p.stage_kb : 1, "B^T"))
      return 1;
  } else {
    VKG_REQUIRE(a->ldb >= a->N, "gemm: ldb %lld < N %d", (long long)a->ldb, a->N);
    if (make_map(dev, &tmB, a->B, a->in_dtype, a->N, a->K, a->ldb, nb0, a->sB0, nb1, a->sB1, b_wide,
                 p.stage_kb * BK, b_wide ? b_groups : 1, "B"))
      return 1;
  }

  out->vec = vec;
  out->total_tiles = (long long)p.tiles_m * p.tiles_n * batch * p.split_k;
  VKG_REQUIRE(out->total_tiles < (1ll << 30), "gemm: too many tiles");
  out->mode = (a->bias ? E_BIAS : 0) | (a->pre ? E_PRE : 0) | (a->act ? E_ACT : 0) |
              (a->dact_z ? E_DACT : 0) | (a->residual ? E_RES : 0) | (a->C2 ? E_C2 : 0) |
              (a->c_dtype == VKG_F16 ? E_F16 : a->c_dtype == VKG_BF16 ? E_BF16 : 0) |
              (a->colsum ? E_COLSUM : 0);
  if (!vec) out->mode = E_GENERIC;
  // write-only epilogues store their tiles through tensor maps over C (and pre); p.C, p.ldc
  // and the batch strides already describe the split-K workspace when K is split
  memset(&out->tmC, 0, sizeof(CUtensorMap));
  memset(&out->tmP, 0, sizeof(CUtensorMap));
  if (dev->tma_store && (out->mode & E_NO_TMA) == 0) {
    const int z1n = p.split_k > 1 ? p.split_k : nb1;
    bool ok_c = false, ok_p = true;
    if (make_out_map(dev, &out->tmC, p.C, p.split_k > 1 ? VKG_F32 : a->c_dtype, p.N, p.M, p.ldc, nb0,
                     p.sC0, z1n, p.sC1, &ok_c))
      return 1;
    if (ok_c && a->pre &&
        make_out_map(dev, &out->tmP, a->pre, VKG_F32, p.N, p.M, p.ldc, nb0, p.sC0, z1n, p.sC1, &ok_p))
      return 1;
    p.tma_store = (ok_c && ok_p) ? 1 : 0;
  }
  return 0;
}

int ensure_attrs(vkg_device* dev) {
  if (dev->gemm_attr_set) return 0;
  VKG_REQUIRE((size_t)SMEM_BYTES <= dev->gemm_smem_optin,
              "gemm needs %d bytes of shared memory, device offers %zu", SMEM_BYTES,
              dev->gemm_smem_optin);
  for (const Specialised& k : kSpecialised)
    VKG_CUDA(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  for (const Specialised& k : kCtaPair)
    VKG_CUDA(cudaFuncSetAttribute(k.fn, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  dev->gemm_attr_set = true;
  return 0;
}

struct ReduceArgs {
  const float4* ws;
  float* C;
  int M, N4;
  long long ldc;
  int splits;
  dim3 grid;
};

ReduceArgs reduce_args(vkg_device* dev, const vkg_gemm_args* a, const GemmParams& p) {
  const long long n4 = (long long)a->M * (a->N / 4);
  return {(const float4*)a->workspace, (float*)a->C, a->M, a->N / 4, (long long)a->ldc, p.split_k,
          dim3(vkg_blocks(n4, 256, (int64_t)dev->sm_count * 8))};
}

int reduce_slices(vkg_device* dev, const vkg_gemm_args* a, const GemmParams& p) {
  if (p.split_k <= 1) return 0;
  const ReduceArgs r = reduce_args(dev, a, p);
  VKG_CUDA(vkg_launch(dev, VKG_K_SMALL | vkg_short_if((long long)r.M * r.N4 <= (1 << 18)), k_splitk_reduce,
                      r.grid, dim3(256), 0, 1, r.ws, r.C, r.M, r.N4, r.ldc, r.splits));
  return vkg_check_launch("splitk_reduce");
}

// A barrier that nothing ever arrives on, waited for with the kernels' own bounded wait and a
// small budget: the error path every device-side wait takes when its partner never shows up
// (flag the abort, record where, return), without a fault and with the context intact.
__global__ void k_wait_selftest(uint32_t* err, long long budget) {
  __shared__ uint64_t bar;
  __shared__ uint32_t abort_flag;
  if (threadIdx.x == 0) {
    abort_flag = 0u;
    mbar_init(smem_u32(&bar), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_wait<true>(smem_u32(&bar), 0, &abort_flag, err, 0x5e1fu, budget);
  }
}

// Adds the per-warp partial column sums a launch left in colsum_scratch: four rows per
// 128-row block the kernel worked on (tile_rows = BM, or 2 * BM for CTA pairs, whose last tile
// may add a block that lies wholly past M and holds zeros).
int finish_colsum(vkg_device* dev, const vkg_gemm_args* a, int tile_rows) {
  if (!a->colsum) return 0;
  const int blocks = ((a->M + tile_rows - 1) / tile_rows) * (tile_rows / BM);
  return vkg_launch_col_sum_final(dev, a->colsum_scratch, a->colsum, a->N, 4 * blocks, 0);
}

}  // namespace

// four partial rows (one per 32-row warp slot) for every 128-row block of the M rows padded
// to the 256-row tiles of a CTA pair
extern "C" int64_t vkg_gemm_colsum_scratch_floats(int M, int N) {
  if (M <= 0 || N <= 0) return 0;
  return (int64_t)4 * 2 * ((M + 2 * BM - 1) / (2 * BM)) * N;
}

extern "C" int64_t vkg_gemm_workspace_bytes(const vkg_gemm_args* a) {
  if (!a || a->M <= 0 || a->N <= 0 || a->K <= 0 || !plain_output(a)) return 0;
  const int split = a->split_k > 0 ? a->split_k : k_slices(a);
  return split > 1 ? (int64_t)split * a->M * a->N * 4 : 0;
}

extern "C" int vkg_selftest_wait_timeout(vkg_device* dev, int64_t budget_cycles) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(budget_cycles > 0 && budget_cycles <= 100000000ll,
              "selftest: budget must be between 1 and 1e8 cycles");
  k_wait_selftest<<<1, 32, 0, dev->stream>>>(dev->err_dev, (long long)budget_cycles);
  return vkg_check_launch("wait_selftest");
}

extern "C" int64_t vkg_gemm_group_table_bytes(int n) {
  return n > 0 ? (int64_t)n * (int64_t)sizeof(GroupEntry) : 0;
}

// Builds the table of a grouped launch in `table` (device memory, 128-byte aligned,
// vkg_gemm_group_table_bytes(n) bytes).  Synchronous: call it outside a stream capture.
extern "C" int vkg_gemm_group_prepare(vkg_device* dev, const vkg_gemm_args* args, int n, void* table,
                                      int cta_pair, int* total_units) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(args && table && total_units && n > 0 && n <= GROUP_MAX,
              "gemm_group: between 1 and %d problems and a table", GROUP_MAX);
  VKG_REQUIRE(((uintptr_t)table & 127) == 0, "gemm_group: table must be 128-byte aligned");
  VKG_REQUIRE(!dev->capturing, "gemm_group: prepare the table before the stream capture begins");
  std::vector<GroupEntry> host(n);
  long long units = 0;
  // CTA-pair tiles (256 x 256) when asked for and every problem has more than one row block
  const bool pair_ok = cta_pair > 0 && dev->sm_count >= 2 &&
                       std::all_of(args, args + n,
                                   [](const vkg_gemm_args& a) { return a.M > BM && a.N >= PAIR_BN / 2; });
  for (int i = 0; i < n; ++i)
    if (check_args(&args[i])) return 1;
  const Tiles tiles = choose_group_tiles(dev, args, n, pair_ok);
  const bool use_pair = tiles.pair;
  for (int i = 0; i < n; ++i) {
    const vkg_gemm_args* a = &args[i];
    const int nb = (a->nb0 > 0 ? a->nb0 : 1) * (a->nb1 > 0 ? a->nb1 : 1);
    VKG_REQUIRE(nb == 1 && a->causal == 0 && !a->bias && !a->pre && !a->act && !a->dact_z &&
                    !a->residual && !a->C2 && !a->colsum && a->c_dtype == VKG_F32 &&
                    (a->alpha == 0.0f || a->alpha == 1.0f),
                "gemm_group: problem %d is not a plain fp32-output, unbatched GEMM", i);
    VKG_REQUIRE(a->in_dtype == args[0].in_dtype, "gemm_group: operand types differ");
    vkg_gemm_args one = *a;
    one.split_k = 1;
    one.workspace = nullptr;
    one.workspace_bytes = 0;
    Problem q;
    if (build_problem(dev, &one, &q, use_pair, tiles.bn, 1, true)) return 1;
    VKG_REQUIRE(q.mode == 0, "gemm_group: problem %d needs 16-byte aligned rows", i);
    memset(&host[i], 0, sizeof(GroupEntry));
    host[i].tmA = q.tmA;
    host[i].tmB = q.tmB;
    host[i].tmC = q.tmC;
    host[i].p = q.p;
    host[i].first_unit = (int)units;
    units += q.total_tiles;
    VKG_REQUIRE(units < (1ll << GROUP_BN_SHIFT), "gemm_group: too many tiles");
  }
  VKG_CUDA(cudaMemcpy(table, host.data(), (size_t)n * sizeof(GroupEntry), cudaMemcpyHostToDevice));
  // a negative count tells vkg_gemm_group_launch that the entries are CTA-pair tiles; otherwise the
  // tile width travels above the count
  *total_units = use_pair ? -(int)units : (int)units + ((tiles.bn / 64 - 1) << GROUP_BN_SHIFT);
  return 0;
}

extern "C" int vkg_gemm_group_launch(vkg_device* dev, const void* table, int n, int total_units) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(table && n > 0 && n <= GROUP_MAX && total_units != 0, "gemm_group: bad arguments");
  if (ensure_attrs(dev)) return 1;
  if (!dev->group_attr_set) {
    VKG_CUDA(cudaFuncSetAttribute(gemm_group_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    VKG_CUDA(cudaFuncSetAttribute(gemm_group_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  SMEM_BYTES));
    dev->group_attr_set = true;
  }
  if (total_units < 0) {
    const int units = -total_units;
    int pairs = vkg_persistent_ctas(dev) / 2;
    if (pairs > units) pairs = units;
    VKG_CUDA(vkg_launch(dev, VKG_K_GEMM_GROUP, gemm_group_pair_kernel, dim3((unsigned)(2 * pairs)), dim3(NUM_THREADS),
                        SMEM_BYTES, 2, static_cast<const GroupEntry*>(table), n, units));
    return vkg_check_launch("gemm_group_pair_kernel");
  }
  const int bn = 64 * ((total_units >> GROUP_BN_SHIFT) + 1);
  total_units &= (1 << GROUP_BN_SHIFT) - 1;
  int ctas = vkg_persistent_ctas(dev) < total_units ? vkg_persistent_ctas(dev) : total_units;
  VKG_CUDA(vkg_launch(dev, VKG_K_GEMM_GROUP | vkg_short_if(total_units <= ctas), gemm_group_kernel,
                      dim3((unsigned)ctas), dim3(NUM_THREADS), SMEM_BYTES, 1,
                      static_cast<const GroupEntry*>(table), n, total_units, bn));
  return vkg_check_launch("gemm_group_kernel");
}

namespace {

// A GEMM ready to launch: which kernel, its launch shape, its parameters and tensor maps.
struct GemmPlan {
  Problem q;
  GemmKernel fn;
  unsigned family, grid;
  bool is_short;      // VKG_SHORT
  int cluster;        // CTAs per thread-block cluster
  int tile_rows;      // rows of C per tile, for the column sums' partial rows
};

int make_plan(vkg_device* dev, const vkg_gemm_args* a, GemmPlan* out) {
  Problem& q = out->q;
  if (check_args(a) || ensure_attrs(dev)) return 1;
  // pairs: only where a pair has at least two row blocks and half a full-width tile to work on,
  // and never for the causal attention shortcuts
  const bool pair_ok = a->causal == 0 && a->M > BM && a->N >= PAIR_BN / 2 && dev->sm_count >= 2 &&
                       (a->tile_n == 0 || a->tile_n == PAIR_BN || a->tile_n == 192) && a->max_ctas == 0 &&
                       a->cta_pair >= 0;
  const bool pair_only = pair_ok && a->cta_pair > 0;
  // the rule's slices, or as many of them as the workspace holds
  int split = a->split_k > 0 ? a->split_k : may_split(a) ? k_slices(a) : 1;
  if (a->split_k <= 0)
    while (split > 1 && (int64_t)split * a->M * a->N * 4 > a->workspace_bytes) --split;
  const int force_bn = pair_only && a->tile_n == 0 ? PAIR_BN : a->tile_n;
  const Tiles t = choose_tiles(dev, a, !pair_only, pair_ok, force_bn, split);
  VKG_REQUIRE(t.us >= 0, "gemm: no tile of %d columns for %d x %d x %d on %d CTAs", a->tile_n, a->M, a->N, a->K,
              a->max_ctas);
  const bool use_pair = t.pair;
  if (build_problem(dev, a, &q, use_pair, t.bn, t.split)) return 1;
  if (use_pair) {
    out->fn = pick(kCtaPair, kNumCtaPair, q.mode);
    long long pairs = vkg_persistent_ctas(dev) / 2;
    if (pairs > q.total_tiles) pairs = q.total_tiles;
    out->family = VKG_K_GEMM_PAIR;
    out->grid = (unsigned)(2 * pairs);
    out->cluster = 2;
    out->tile_rows = 2 * BM;
  } else {
    out->fn = pick(kSpecialised, kNumSpecialised, q.mode);
    long long ctas = a->max_ctas > 0 ? a->max_ctas : vkg_persistent_ctas(dev);
    if (ctas > q.total_tiles) ctas = q.total_tiles;
    out->family = VKG_K_GEMM;
    out->grid = (unsigned)ctas;
    out->cluster = 1;
    out->tile_rows = BM;
  }
  // no CTA works on a second tile, or it is over soon all the same
  out->is_short = q.total_tiles * out->cluster <= (long long)out->grid || t.us < PL_SHORT_US;
  return 0;
}

// Eager launches go through a small executable graph per launch shape (single CTAs or pairs, with
// or without the K-slice reduction): stamp, kernel(s), stamp.  The kernel nodes get the plan's
// parameters before each launch (0.2 us), so one graph serves every call of its shape.  Launch to
// result on B200, for a kernel of 1 us: 6.6 us, against 15.6 us for event, launch, event, wait.
struct EagerGraph {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  cudaGraphNode_t gemm = nullptr, reduce = nullptr;
};

// Plans by argument block.  A plan holds addresses, shapes and launch choices and nothing that
// lives behind the pointers, so it stays valid for as long as the same arguments are passed; an
// eager loop over the same operands pays for planning and four tensor maps once (about 3 us).
// Bounded: emptied when full.
struct PlanCache {
  static constexpr size_t LIMIT = 256;
  std::mutex mu;
  std::unordered_map<std::string, GemmPlan> plans;
  std::mutex eager_mu;
  EagerGraph eager[3][2][2];  // by CTAs per cluster, with and without the reduction, overlapping or not
};

int find_plan(vkg_device* dev, const vkg_gemm_args* a, GemmPlan* out) {
  const int tuning[4] = {vkg_persistent_ctas(dev), dev->tma_store ? 1 : 0, dev->pair_min_waves_x10,
                         dev->pair192 ? 1 : 0};
  std::string key(reinterpret_cast<const char*>(a), sizeof(*a));
  key.append(reinterpret_cast<const char*>(tuning), sizeof(tuning));
  PlanCache* cache = static_cast<PlanCache*>(dev->gemm_plans);
  {
    std::lock_guard<std::mutex> lock(cache->mu);
    auto it = cache->plans.find(key);
    if (it != cache->plans.end()) {
      *out = it->second;
      return 0;
    }
  }
  if (make_plan(dev, a, out)) return 1;
  std::lock_guard<std::mutex> lock(cache->mu);
  if (cache->plans.size() >= PlanCache::LIMIT) cache->plans.clear();
  cache->plans.emplace(std::move(key), *out);
  return 0;
}

int launch_plan(vkg_device* dev, const vkg_gemm_args* a, const GemmPlan& pl) {
  const Problem& q = pl.q;
  VKG_CUDA(vkg_launch(dev, pl.family | vkg_short_if(pl.is_short), pl.fn, dim3(pl.grid), dim3(NUM_THREADS),
                      SMEM_BYTES, pl.cluster, q.tmA, q.tmB, q.tmC, q.tmP, q.p));
  if (vkg_check_launch("gemm")) return 1;
  if (reduce_slices(dev, a, q.p)) return 1;
  return finish_colsum(dev, a, pl.tile_rows);
}

}  // namespace

extern "C" int vkg_gemm(vkg_device* dev, const vkg_gemm_args* a) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(a, "null gemm args");
  GemmPlan pl;
  if (find_plan(dev, a, &pl)) return 1;
  return launch_plan(dev, a, pl);
}

namespace {

int eager_graph_build(vkg_device* dev, const vkg_gemm_args* a, const GemmPlan& pl, EagerGraph* out) {
  const int pdl = dev->pdl;
  if (pdl < 0) dev->pdl = 1;     // stamps and kernel overlap, whatever size the nodes are reused for
  VKG_CUDA(cudaStreamBeginCapture(dev->stream, cudaStreamCaptureModeThreadLocal));
  const int bad = vkg_stamp_begin(dev, &dev->timer) || launch_plan(dev, a, pl) || vkg_stamp_end(dev, &dev->timer);
  cudaGraph_t g = nullptr;
  const cudaError_t e = cudaStreamEndCapture(dev->stream, &g);
  dev->pdl = pdl;
  if (bad) {
    if (g) cudaGraphDestroy(g);
    return 1;
  }
  VKG_REQUIRE(e == cudaSuccess && g, "eager gemm: capture failed: %s", cudaGetErrorString(e));
  out->graph = g;
  cudaGraphNode_t nodes[8];
  size_t n = 8;
  VKG_CUDA(cudaGraphGetNodes(g, nodes, &n));
  for (size_t i = 0; i < n; ++i) {
    cudaKernelNodeParams kp;
    VKG_CUDA(cudaGraphKernelNodeGetParams(nodes[i], &kp));
    if (kp.func == (void*)k_splitk_reduce) out->reduce = nodes[i];
    else if (!vkg_is_stamp_kernel(kp.func)) out->gemm = nodes[i];
  }
  VKG_REQUIRE(out->gemm, "eager gemm: no kernel node");
  VKG_CUDA(cudaGraphInstantiate(&out->exec, g, 0));
  return 0;
}

int eager_graph_launch(vkg_device* dev, const vkg_gemm_args* a, const GemmPlan& pl, EagerGraph* eg) {
  const Problem& q = pl.q;
  cudaKernelNodeParams kp;
  memset(&kp, 0, sizeof(kp));
  void* args[] = {(void*)&q.tmA, (void*)&q.tmB, (void*)&q.tmC, (void*)&q.tmP, (void*)&q.p};
  kp.func = (void*)pl.fn;
  kp.gridDim = dim3(pl.grid);
  kp.blockDim = dim3(NUM_THREADS);
  kp.sharedMemBytes = SMEM_BYTES;
  kp.kernelParams = args;
  VKG_CUDA(cudaGraphExecKernelNodeSetParams(eg->exec, eg->gemm, &kp));
  if (eg->reduce) {
    ReduceArgs r = reduce_args(dev, a, q.p);
    void* rargs[] = {&r.ws, &r.C, &r.M, &r.N4, &r.ldc, &r.splits};
    kp.func = (void*)k_splitk_reduce;
    kp.gridDim = r.grid;
    kp.blockDim = dim3(256);
    kp.sharedMemBytes = 0;
    kp.kernelParams = rargs;
    VKG_CUDA(cudaGraphExecKernelNodeSetParams(eg->exec, eg->reduce, &kp));
  }
  VKG_CUDA(cudaGraphLaunch(eg->exec, dev->stream));
  return 0;
}

}  // namespace

extern "C" int vkg_gemm_run(vkg_device* dev, const vkg_gemm_args* a, int repeat, double* seconds) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(a && repeat >= 0, "gemm_run: bad arguments");
  GemmPlan pl;
  if (find_plan(dev, a, &pl)) return 1;
  if (repeat == 1 && !a->colsum && !dev->capturing) {
    PlanCache* cache = static_cast<PlanCache*>(dev->gemm_plans);
    std::lock_guard<std::mutex> lock(cache->eager_mu);     // the graphs and the timer stamp are shared
    EagerGraph& eg = cache->eager[pl.cluster][pl.q.p.split_k > 1 ? 1 : 0][dev->pdl ? 1 : 0];
    if (!eg.exec && eager_graph_build(dev, a, pl, &eg)) return 1;
    if (eager_graph_launch(dev, a, pl, &eg)) return 1;
    dev->timer.launched++;
    return vkg_stamp_finish(dev, &dev->timer, "gemm", seconds);
  }
  if (vkg_timer_begin(dev)) return 1;
  for (int i = 0; i < repeat; ++i)
    if (launch_plan(dev, a, pl)) return 1;
  return vkg_timer_end(dev, seconds);
}

void* vkg_gemm_plans_create() { return new PlanCache(); }
void vkg_gemm_plans_destroy(void* cache) {
  PlanCache* c = static_cast<PlanCache*>(cache);
  if (!c) return;
  for (auto& plane : c->eager)
    for (auto& row : plane)
      for (EagerGraph& eg : row) {
        if (eg.exec) cudaGraphExecDestroy(eg.exec);
        if (eg.graph) cudaGraphDestroy(eg.graph);
      }
  delete c;
}
