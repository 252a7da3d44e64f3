// Fused causal attention for sm_100a, head dimension 64: replaces the reference's
// per-layer chain  QK^T matmul -> attn_softmax -> PV matmul  (transformer.py:144-155)
// and its backward chain (transformer.py:167-182) without ever writing the T x T score,
// probability or gradient tensors to HBM.
//
// Forward, one CTA per (128-query tile, head, sequence), 320 threads, two CTAs per SM:
//   warp 0      TMA producer: Q once, then the K and V tiles
//   warp 1      TMEM allocation + tcgen05.mma issue (the warp runs converged, one elected lane
//               per instruction)
//   warps 2..9  softmax: TMEM lane = query row; two warps share a lane quarter, each takes 64
//               of a tile's 128 keys, so a thread owns half of one row
// Two kernels.  attn_fwd1_kernel (the default) makes one pass: S = Q K^T once per key tile,
// P~ = exp2(S c - m) against a running reference maximum m that is moved -- and O~ and the row
// sum rescaled -- only when a tile exceeds it by more than 2^8.  attn_fwd_kernel makes two:
//   pass 1  S = Q K^T  -> row maximum m only (no exponentials)
//   pass 2  S again, P~ = exp2(S c - m), O~ += P~ V, no rescaling at all
// (QK^T has K = 64, so doing it twice costs little: 45 vs 37 us per layer at 8 x 1024 x 12.)
// In both, P~ is rounded to fp16 -- into tensor memory in the one-pass kernel, where P~ V reads
// it as the A operand, into swizzled shared memory in the two-pass one --, O~ accumulates in
// TMEM, the row sum l of the UN-rounded P~ is kept in fp32, and O = O~ / l when the tile is
// stored.
// Backward: two persistent kernels, the dQ kernel (which also forms delta = rowsum(dO * O))
// and the dK / dV kernel; their comments are beside them.
// Rounding points against the reference: it rounds the NORMALISED probability P = P~ / l to
// fp16 before P V (tkernels.py:123); here the un-normalised P~ (in (0, 1], the row's largest
// entry exactly 1) is rounded and 1 / l is applied to the fp32 accumulator, so O carries the
// same relative rounding per product and one division less per score.  The backward kernels
// rebuild the normalised P from the saved log-sum-exp and round that, as the reference does
// (tkernels.py:123, 183); O, dQ, dK, dV are stored fp16 as there (tkernels.py:284, 228-230).
// Every wait on a barrier is bounded (see tcgen05.cuh); a wait that gives up flags the error word,
// all roles leave their loops, TMEM is freed and the CTA returns.  The backward's request for registers
// has no limit; the host makes sure that it can be met.
#include "common.cuh"
#include "tcgen05.cuh"

namespace {

using namespace tc05;

constexpr int FA_T = 128;          // query / key tile
constexpr int FA_HD = 64;          // head dimension
constexpr int FA_TILE_BYTES = FA_T * FA_HD * 2;  // 16 KB: one 128 x 64 fp16 tile, 128 B rows
constexpr int FA_THREADS = 320;      // producer + MMA + eight softmax warps
constexpr int FA_SOFTMAX_WARPS = 8;
constexpr float LOG2E = 1.4426950408889634f;
// The softmax warps' waits suspend (mbarrier.try_wait with a time hint); the producer's and the
// MMA warps', which sit on the critical chain, poll.  Polling in the softmax warps too measured
// the same to 1 us per layer.
constexpr bool SM_SPIN = false;

struct AttnParams {
  int B, T, H, D;
  int nqt;                 // query tiles per sequence
  float cscale;            // softmax scale * log2(e)
  float scale;
  const uint32_t* seg;     // optional packed-sample starts (b*T + t)
  int skip_tiles;          // packed, and worth looking for tiles that are wholly masked
  __half* out;             // forward: O, head-merged (rows, D)
  float* lse2;             // (B*H, T): row log2-sum-exp of the scaled scores
  const float* delta;      // backward: rowsum(dO * O), (B*H, T); the dQ kernel writes it (delta_out),
  float* delta_out;        // the dK / dV kernel, launched after it, reads it
  __half* dqkv;            // backward: (rows, 3D)
  float* colsum;           // backward, optional: [B * nqt * 4][3D] partial column sums of dqkv
  uint32_t* err;
};

// forward shared memory map (offsets from a 1024-aligned base)
constexpr int FW_Q = 0;
constexpr int FW_K = FW_Q + FA_TILE_BYTES;            // two K stages
constexpr int FW_V = FW_K + 2 * FA_TILE_BYTES;        // one V stage
constexpr int FW_P = FW_V + FA_TILE_BYTES;            // P: two 64-key blocks of 128 rows x 128 B
constexpr int FW_BAR = FW_P + 2 * FA_TILE_BYTES;
constexpr int FW_XCHG = FW_BAR + 256;                 // row statistics exchange: [2][128] floats; the
                                                      // one-pass kernel: [2][2][128] tagged 8-byte
                                                      // slots, then [2][128] floats
constexpr int FW_SMEM = FW_XCHG + 4096 + 1024 + 1024;

// P and dS tiles use the 128B-swizzled layout of TMA and the UMMA descriptors: 16-byte
// piece c8 (8 keys) of row r of a 64-key block sits at r * 128 + ((c8 ^ (r & 7)) << 4).

// Packed batches: the smallest sample start among a query tile's rows, taken by one warp.  Key tiles
// that lie wholly before it are masked for every row; what they would add is exactly zero, so the
// kernels pass over them.  Nothing is assumed about the order of the starts.
__device__ __forceinline__ int tile_first_start(const uint32_t* seg, int q0, int T, int lane) {
  uint32_t v = 0x7fffffffu;
#pragma unroll
  for (int i = 0; i < FA_T / 32; ++i) {
    const int q = q0 + i * 32 + lane;
    if (q < T) v = min(v, seg[q]);
  }
  return (int)__reduce_min_sync(0xffffffffu, v);
}
constexpr int SEG_ITEMS = 64, SEG_TILES = 32;      // items of a CTA, tiles of a sequence this is done for
// Reading the starts takes a kernel half a microsecond before its first load.  From three tiles to a
// sequence on it saves more (2 x 700 tokens, 6 heads, samples of 170: forward 17.5 -> 14.1 us); one or
// two tiles rarely have one to pass over.
int skip_tiles(const uint32_t* seg, int nqt) { return seg && nqt > 2 && nqt <= SEG_TILES; }

// What the causal rule and the sample starts leave of a warp's block of nq queries from q0 on and nk keys
// from k0 on, the starts lying in st_min .. st_max: everything, some of it (tested element by element),
// or nothing (no arithmetic at all).  Packed batches only: with the causal rule alone, where one tile in
// several has such blocks, the extra paths measured more than they saved (8 x 1024 x 12, dK / dV: 49 -> 63 us).
enum : int { BLOCK_ALL, BLOCK_SOME, BLOCK_NONE };
__device__ __forceinline__ int block_class(int q0, int nq, int k0, int nk, int st_min, int st_max) {
  if (k0 > q0 + nq - 1 || st_min > k0 + nk - 1) return BLOCK_NONE;
  return k0 + nk - 1 <= q0 && st_max <= k0 ? BLOCK_ALL : BLOCK_SOME;
}

// Row maximum over this thread's 64 raw scores of one key tile.  MASK adds the causal /
// packed-sample test and is compiled only into the tiles that need it.
template <bool MASK>
__device__ __forceinline__ float fwd_max_tile(const uint32_t (&r)[64], int key0, int qi, int st, float m) {
#pragma unroll
  for (int e = 0; e < 64; ++e) {
    if (MASK) {
      const int key = key0 + e;
      if (key > qi || key < st) continue;
    }
    m = fmaxf(m, __uint_as_float(r[e]));
  }
  return m;
}

// P = exp2(s * cscale - m) for this thread's 64 scores, rounded to fp16 into the swizzled
// row `prow` (x = row & 7); returns the fp32 sum of the row's part.
template <bool MASK>
__device__ __forceinline__ float fwd_p_tile(const uint32_t (&r)[64], int key0, int qi, int st, float cscale,
                                         float nm, uint8_t* prow, uint32_t x) {
  float l = 0.f;
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    __half2 hv[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float pv[2];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int idx = u * 8 + 2 * e + w;
        float pr = vkg_ex2(fmaf(__uint_as_float(r[idx]), cscale, nm));
        if (MASK) {
          const int key = key0 + idx;
          if (key > qi || key < st) pr = 0.f;
        }
        pv[w] = pr;
      }
      l += pv[0] + pv[1];
      hv[e] = __floats2half2_rn(pv[0], pv[1]);
    }
    *reinterpret_cast<uint4*>(prow + (((uint32_t)u ^ x) << 4)) = *reinterpret_cast<uint4*>(hv);
  }
  return l;
}

// The same exponentials for a P~ that stays in tensor memory: the fp16 pairs (keys 2i, 2i + 1)
// replace r[i], ready for tcgen05.st; returns the fp32 sum of the un-rounded values.
template <bool MASK>
__device__ __forceinline__ float fwd_p_pack(uint32_t (&r)[64], int key0, int qi, int st, float cscale,
                                            float nm) {
  float l = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    float pv[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      float pr = vkg_ex2(fmaf(__uint_as_float(r[2 * i + w]), cscale, nm));
      if (MASK) {
        const int key = key0 + 2 * i + w;
        if (key > qi || key < st) pr = 0.f;
      }
      pv[w] = pr;
    }
    l += pv[0] + pv[1];
    const __half2 h = __floats2half2_rn(pv[0], pv[1]);
    r[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  return l;
}

// Store a warp's block of 32 rows x NU 16-byte groups (lane = row, v[u] = group u of the row)
// to global rows of `pitch` bytes so that every store instruction writes whole contiguous row
// segments: the block goes through the warp's private staging area (32 x NU x 16 bytes, XOR
// swizzled so both passes are conflict-free) and comes back with 32 / NU rows per instruction.
// One row per lane (128-byte rows 4608 bytes apart for a 768-wide model) measured 1.5 us per
// item on the softmax warps' critical path.  rows_ok = how many of the 32 rows exist.
template <int NU>
__device__ __forceinline__ void warp_store_rows(const uint4 (&v)[NU], uint8_t* stage, int lane,
                                                uint8_t* dst_row0, size_t pitch, int rows_ok) {
  static_assert(NU == 4 || NU == 8, "64- or 128-byte row segments");
#pragma unroll
  for (int u = 0; u < NU; ++u)
    *reinterpret_cast<uint4*>(stage + lane * (NU * 16) + ((u ^ (lane & (NU - 1))) << 4)) = v[u];
  __syncwarp();
  constexpr int RPI = 32 / NU;        // rows per store instruction
  const int u = lane % NU;
#pragma unroll
  for (int i = 0; i < NU; ++i) {
    const int row = i * RPI + lane / NU;
    const uint4 x = *reinterpret_cast<const uint4*>(stage + row * (NU * 16) + ((u ^ (row & (NU - 1))) << 4));
    if (row < rows_ok) *reinterpret_cast<uint4*>(dst_row0 + (size_t)row * pitch + u * 16) = x;
  }
  __syncwarp();
}

__global__ void __launch_bounds__(FA_THREADS, 2)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tm, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + FW_BAR;
  // barriers: 0 q_full, 1-2 k_full, 3-4 k_empty, 5 v_full, 6 v_empty, 7 s_full, 8 s_free,
  //           9 p_full, 10 p_free, 11 o_full
  auto B_ = [bar](int i) { return bar + 8u * i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + FW_BAR + 128);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(gbase + FW_BAR + 136);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int HB = p.H * p.B;
  const int qt = p.nqt - 1 - (int)(blockIdx.x / HB);   // heaviest query tiles first
  const int hb = blockIdx.x % HB;
  const int h = hb % p.H, b = hb / p.H;
  const int q0 = qt * FA_T;
  const int nj = qt + 1;                                 // key tiles 0..qt
  const int row0 = b * p.T;                              // first row of this sequence

  pdl_trigger();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm);
    for (int i = 0; i < 12; ++i) mbar_init(B_(i), (i == 8 || i == 9) ? FA_SOFTMAX_WARPS : 1);
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 256);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();      // the projection that wrote qkv has completed
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tO = tmem + 128;

  if (warp == 0) {
    if (lane == 0) {
      bool ok = true;
      mbar_expect_tx(B_(0), FA_TILE_BYTES);
      tma_load_2d(base + FW_Q, &tm, B_(0), h * FA_HD, row0 + q0);
      int it = 0;
      for (int pass = 0; pass < 2 && ok; ++pass) {
        for (int j = 0; j < nj && ok; ++j, ++it) {
          const int s = it & 1;
          ok = mbar_wait<true>(B_(3 + s), ((it >> 1) & 1) ^ 1u, abort_flag, p.err, 0x1100u + s);
          if (!ok) break;
          mbar_expect_tx(B_(1 + s), FA_TILE_BYTES);
          tma_load_2d(base + FW_K + s * FA_TILE_BYTES, &tm, B_(1 + s), p.D + h * FA_HD,
                      row0 + j * FA_T);
          if (pass == 1) {
            ok = mbar_wait<true>(B_(6), (j & 1) ^ 1u, abort_flag, p.err, 0x1200u);
            if (!ok) break;
            mbar_expect_tx(B_(5), FA_TILE_BYTES);
            tma_load_2d(base + FW_V, &tm, B_(5), 2 * p.D + h * FA_HD, row0 + j * FA_T);
          }
        }
      }
    }
  } else if (warp == 1) {
    // the whole warp runs this converged; one elected lane issues each tcgen05 instruction
    const uint32_t idesc_s = make_idesc(0, 0, 0, FA_T);     // Q K^T: both K-major, N = 128 keys
    const uint32_t idesc_o = make_idesc(0, 0, 1, FA_HD);    // P V: P K-major, V MN-major, N = 64
    bool ok = mbar_wait_warp<true>(B_(0), 0, abort_flag, p.err, 0x2000u);
    // descriptor halves (tcgen05.cuh): start address and leading offset in the low word
    const uint32_t d_hi = smem_desc_hi(1024);
    const uint32_t q_lo = smem_desc_lo(base + FW_Q, 16), k_lo = smem_desc_lo(base + FW_K, 16);
    const uint32_t p_lo = smem_desc_lo(base + FW_P, 16), v_lo = smem_desc_lo(base + FW_V, 8192);
    // S number n (n counts both passes): wait for its K stage and for the softmax warps
    // to have pulled the previous S out of TMEM, then issue Q K^T.
    auto issue_s = [&](int n) -> bool {
      const int s = n & 1;
      if (!(mbar_wait_warp<true>(B_(1 + s), (n >> 1) & 1, abort_flag, p.err, 0x2100u + s) &&
            mbar_wait_warp<true>(B_(8), (n & 1) ^ 1u, abort_flag, p.err, 0x2200u)))
        return false;
      tcgen05_fence_after();
      umma_f16_chain<4>(tS, q_lo, 2, k_lo + (uint32_t)s * (FA_TILE_BYTES >> 4), 2, d_hi, idesc_s, 0u);
      umma_commit_one(B_(3 + s));   // K stage free once these retire
      umma_commit_one(B_(7));       // S ready
      return true;
    };
    // pass 1: S only.  Pass 2 is software-pipelined: S(j+1) is issued before P(j) V, so
    // the tensor core works on the next scores while the softmax warps finish P(j).
    int n = 0;
    for (; n < nj && ok; ++n) ok = issue_s(n);
    if (ok) ok = issue_s(n++);
    for (int j = 0; j < nj && ok; ++j) {
      if (j + 1 < nj) {
        ok = issue_s(n++);
        if (!ok) break;
      }
      ok = mbar_wait_warp<true>(B_(9), j & 1, abort_flag, p.err, 0x2300u) &&
           mbar_wait_warp<true>(B_(5), j & 1, abort_flag, p.err, 0x2400u);
      if (!ok) break;
      tcgen05_fence_after();
      // P: two 64-key blocks, K-major; V: MN-major, 16 keys = two 8-row groups further down
      umma_f16_chain<4>(tO, p_lo, 2, v_lo, 128, d_hi, idesc_o, j ? 1u : 0u);
      umma_f16_chain<4>(tO, p_lo + (FA_TILE_BYTES >> 4), 2, v_lo + 4 * 128, 128, d_hi, idesc_o, 1u);
      umma_commit_one(B_(6));     // V free
      umma_commit_one(B_(10));    // P free
    }
    if (ok) umma_commit_one(B_(11));
  } else {
    // Softmax: two warps per TMEM lane quarter; `half` picks which 64 of the tile's 128
    // keys this warp handles.  Each thread owns one query row of its half.
    const int half = (warp - 2) >> 2;
    const int qr = (warp & 3) * 32 + lane;      // row within the tile = TMEM lane
    const int qi = q0 + qr;                     // query index in the sequence
    const bool q_ok = qi < p.T;
    const int st = (p.seg && q_ok) ? (int)p.seg[row0 + qi] : 0;
    const uint32_t t_lane = ((uint32_t)((warp & 3) * 32)) << 16;
    float* xchg = reinterpret_cast<float*>(gbase + FW_XCHG);   // [2][128] row statistics
    float m = -1e30f, l = 0.f;
    bool ok = true;
    int it = 0;
    // pass 1: row maximum of the scaled scores (no exponentials)
    for (int j = 0; j < nj && ok; ++j, ++it) {
      ok = mbar_wait_warp<SM_SPIN>(B_(7), it & 1, abort_flag, p.err, 0x3100u);
      if (!ok) break;
      tcgen05_fence_after();
      const bool need_mask = (j == qt) || (p.seg != nullptr);
      uint32_t r[64];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(tS + t_lane + half * 64 + c * 16, r + c * 16);
      tmem_wait_ld();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(8));        // S may be overwritten
      // the scale is positive, so the maximum of the raw scores is enough here
      if (need_mask) m = fwd_max_tile<true>(r, j * FA_T + half * 64, qi, st, m);
      else m = fwd_max_tile<false>(r, 0, 0, 0, m);
    }
    xchg[half * 128 + qr] = m;
    asm volatile("bar.sync 1, 256;" ::: "memory");   // the eight softmax warps
    m = fmaxf(xchg[qr], xchg[128 + qr]) * p.cscale;  // row maximum of the scaled scores
    const float nm = -m;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    // pass 2: P = exp2(t - m) rounded to fp16 (normalised by 1/l at the very end), l in fp32
    for (int j = 0; j < nj && ok; ++j, ++it) {
      ok = mbar_wait_warp<SM_SPIN>(B_(7), it & 1, abort_flag, p.err, 0x3150u);
      if (!ok) break;
      tcgen05_fence_after();
      const bool need_mask = (j == qt) || (p.seg != nullptr);
      uint32_t r[64];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(tS + t_lane + half * 64 + c * 16, r + c * 16);
      tmem_wait_ld();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(8));
      ok = mbar_wait_warp<SM_SPIN>(B_(10), (j & 1) ^ 1u, abort_flag, p.err, 0x3200u);   // P buffer free
      if (!ok) break;
      uint8_t* prow = gbase + FW_P + half * FA_TILE_BYTES + qr * 128;
      if (need_mask) l += fwd_p_tile<true>(r, j * FA_T + half * 64, qi, st, p.cscale, nm, prow, qr & 7);
      else l += fwd_p_tile<false>(r, 0, 0, 0, p.cscale, nm, prow, qr & 7);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(9));        // this warp's part of P is in shared memory
    }
    xchg[half * 128 + qr] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l = xchg[qr] + xchg[128 + qr];
    const float inv_l = 1.0f / l;               // l >= 1: key == query is always valid
    if (half == 0 && q_ok) p.lse2[(size_t)(b * p.H + h) * p.T + qi] = m + log2f(l);
    if (ok) ok = mbar_wait_warp<SM_SPIN>(B_(11), 0, abort_flag, p.err, 0x3300u);
    if (ok) {
      tcgen05_fence_after();
      uint32_t r[32];                            // this half's 32 of the 64 output columns
      tmem_ld16(tO + t_lane + half * 32, r);
      tmem_ld16(tO + t_lane + half * 32 + 16, r + 16);
      tmem_wait_ld();
      {
        uint4 hv[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          __half2 h2[4];
#pragma unroll
          for (int e = 0; e < 4; ++e)
            h2[e] = __floats2half2_rn(__uint_as_float(r[u * 8 + 2 * e]) * inv_l,
                                      __uint_as_float(r[u * 8 + 2 * e + 1]) * inv_l);
          hv[u] = *reinterpret_cast<uint4*>(h2);
        }
        // every product has retired (o_full), so the P buffer serves as the staging area
        const int q_w = q0 + (warp & 3) * 32;
        __half* dst = p.out + (size_t)(row0 + q_w) * p.D + h * FA_HD + half * 32;
        warp_store_rows<4>(hv, gbase + FW_P + (warp - 2) * 2048, lane, reinterpret_cast<uint8_t*>(dst),
                           (size_t)p.D * 2, p.T - q_w);
      }
    }
  }

  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// ---- forward, one pass ------------------------------------------------------------------
//
// The same CTA shape and roles, but every S = Q K^T is computed once: the softmax warps keep a
// running reference maximum m per row, P~ = exp2(S c - m) goes to the tensor core as before,
// and O~ and the row sum l are rescaled only when a tile's row maximum exceeds the reference by
// more than 2^8 (then the warps multiply their columns of O~ in TMEM by exp2(m_old - m_new)).
// With the threshold P~ stays below 256, well inside fp16, and its relative rounding is that of
// the two-pass kernel; for ordinary score ranges no rescale ever runs.  The two warps that share
// a row (64 keys each) exchange their tile maxima through shared memory with a tagged slot and
// a bounded poll -- no named barrier inside the loop, so an aborting warp cannot strand its
// partner.  The rescale sits between "P V of the previous tile has retired" (the wait that
// guards the P buffer anyway) and this warp's arrival on p_full, so it needs no barrier of its
// own: O~ is quiet exactly there.
// P~ in tensor memory leaves shared memory for three stages of K and two of V.  With two and one, a
// single V stage made every load (0.8 us) wait for the product before it, and the producer, which
// issues loads in order, held K of the next tile behind that V: a tile took load + product, 1.45 us,
// wherever one CTA has an SM to itself.
constexpr float FW1_LAZY = 8.0f;      // log2 of the largest P~ the running reference allows
constexpr int F1_K_STAGES = 3, F1_V_STAGES = 2;
constexpr int F1_K = FW_K, F1_V = F1_K + F1_K_STAGES * FA_TILE_BYTES;
constexpr int F1_OUT = F1_V;          // output staging, once every product has retired
static_assert(F1_V + F1_V_STAGES * FA_TILE_BYTES <= FW_BAR, "one-pass forward: shared memory");

template <bool PACKED>
__global__ void __launch_bounds__(FA_THREADS, 2)
attn_fwd1_kernel(const __grid_constant__ CUtensorMap tm, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + FW_BAR;
  // barriers: 0 q_full, 1-2 v_full, 3-4 v_empty, 5-7 k_full, 12-14 k_empty, 15 s_full, 8 s_free,
  //           9 p_full, 10 p_free, 11 o_full
  auto B_ = [bar](int i) { return bar + 8u * i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + FW_BAR + 128);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(gbase + FW_BAR + 136);
  // [parity][half][row] (tag, value) pairs for the per-tile maxima; the final row sums reuse it
  volatile unsigned long long* xslot = reinterpret_cast<volatile unsigned long long*>(gbase + FW_XCHG);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int HB = p.H * p.B;
  const int qt = p.nqt - 1 - (int)(blockIdx.x / HB);   // heaviest query tiles first
  const int hb = blockIdx.x % HB;
  const int h = hb % p.H, b = hb / p.H;
  const int q0 = qt * FA_T;
  const int nj = qt + 1;
  const int row0 = b * p.T;

  pdl_trigger();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm);
    for (int i = 0; i < 16; ++i) mbar_init(B_(i), (i == 8 || i == 9) ? FA_SOFTMAX_WARPS : 1);
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  for (int i = threadIdx.x; i < 2 * 2 * FA_T; i += blockDim.x) xslot[i] = 0ull;   // tag 0 = empty
  if (warp == 1) tmem_alloc(tmem_slot, 256);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();
  int j0 = 0;                      // first key tile that counts
  if (PACKED && p.skip_tiles) {
    volatile int* slot = reinterpret_cast<volatile int*>(gbase + FW_BAR + 144);
    if (warp == 0) {
      const int st = tile_first_start(p.seg + row0, q0, p.T, lane);
      if (lane == 0) *slot = min(st / FA_T, qt);
    }
    __syncthreads();
    j0 = *slot;
  }
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tO = tmem + 128, tP = tmem + 192;   // P~: 128 keys, two per column

  if (warp == 0) {
    if (lane == 0) {
      mbar_expect_tx(B_(0), FA_TILE_BYTES);
      tma_load_2d(base + FW_Q, &tm, B_(0), h * FA_HD, row0 + q0);
      int ks = 0;
      uint32_t kph = 0;
      for (int j = j0, n = 0; j < nj; ++j, ++n) {
        if (!mbar_wait<true>(B_(12 + ks), kph ^ 1u, abort_flag, p.err, 0x6100u + ks)) break;
        mbar_expect_tx(B_(5 + ks), FA_TILE_BYTES);
        tma_load_2d(base + F1_K + ks * FA_TILE_BYTES, &tm, B_(5 + ks), p.D + h * FA_HD, row0 + j * FA_T);
        if (++ks == F1_K_STAGES) {
          ks = 0;
          kph ^= 1u;
        }
        const int vs = n & 1;
        if (!mbar_wait<true>(B_(3 + vs), ((n >> 1) & 1) ^ 1u, abort_flag, p.err, 0x6200u + vs)) break;
        mbar_expect_tx(B_(1 + vs), FA_TILE_BYTES);
        tma_load_2d(base + F1_V + vs * FA_TILE_BYTES, &tm, B_(1 + vs), 2 * p.D + h * FA_HD, row0 + j * FA_T);
      }
    }
  } else if (warp == 1) {
    // the whole warp runs this converged; one elected lane issues each tcgen05 instruction
    const uint32_t idesc_s = make_idesc(0, 0, 0, FA_T);
    const uint32_t idesc_o = make_idesc(0, 0, 1, FA_HD);
    bool ok = mbar_wait_warp<true>(B_(0), 0, abort_flag, p.err, 0x7000u);
    // descriptor halves (tcgen05.cuh): start address and leading offset in the low word
    const uint32_t d_hi = smem_desc_hi(1024);
    const uint32_t q_lo = smem_desc_lo(base + FW_Q, 16), k_lo = smem_desc_lo(base + F1_K, 16);
    const uint32_t v_lo = smem_desc_lo(base + F1_V, 8192);
    int ks = 0;
    uint32_t kph = 0;
    auto issue_s = [&](int n) -> bool {
      if (!(mbar_wait_warp<true>(B_(5 + ks), kph, abort_flag, p.err, 0x7100u + ks) &&
            mbar_wait_warp<true>(B_(8), (n & 1) ^ 1u, abort_flag, p.err, 0x7200u)))
        return false;
      tcgen05_fence_after();
      umma_f16_chain<4>(tS, q_lo, 2, k_lo + (uint32_t)ks * (FA_TILE_BYTES >> 4), 2, d_hi, idesc_s, 0u);
      umma_commit_one(B_(12 + ks));   // K stage free once these retire
      umma_commit_one(B_(15));        // S ready
      if (++ks == F1_K_STAGES) {
        ks = 0;
        kph ^= 1u;
      }
      return true;
    };
    int n = 0;
    if (ok) ok = issue_s(n++);
    for (int j = 0; j0 + j < nj && ok; ++j) {
      if (j0 + j + 1 < nj) {     // the next scores first: the tensor core works while P(j) forms
        ok = issue_s(n++);
        if (!ok) break;
      }
      ok = mbar_wait_warp<true>(B_(9), j & 1, abort_flag, p.err, 0x7300u) &&
           mbar_wait_warp<true>(B_(1 + (j & 1)), (j >> 1) & 1, abort_flag, p.err, 0x7400u);
      if (!ok) break;
      tcgen05_fence_after();
      // P~ from tensor memory; V: MN-major, 16 keys = two 8-row groups further down
      umma_f16_ts_chain<8>(tO, tP, v_lo + (uint32_t)(j & 1) * (FA_TILE_BYTES >> 4), 128, d_hi, idesc_o,
                           j ? 1u : 0u);
      umma_commit_one(B_(3 + (j & 1)));     // V stage free
      umma_commit_one(B_(10));    // P free, and O~ quiet until the next p_full
    }
    if (ok) umma_commit_one(B_(11));
  } else {
    const int half = (warp - 2) >> 2;
    const int qr = (warp & 3) * 32 + lane;      // row within the tile = TMEM lane
    const int qi = q0 + qr;
    const bool q_ok = qi < p.T;
    const int st = (PACKED && q_ok) ? (int)p.seg[row0 + qi] : 0;
    const int st_min = PACKED ? __reduce_min_sync(0xffffffffu, st) : 0;
    const int st_max = PACKED ? __reduce_max_sync(0xffffffffu, st) : 0;
    const uint32_t t_lane = ((uint32_t)((warp & 3) * 32)) << 16;
    float m_ref = -1e30f, l = 0.f;              // reference maximum (scaled units), row sum
    bool ok = true;
    for (int n = 0; j0 + n < nj && ok; ++n) {
      const int j = j0 + n;
      ok = mbar_wait_warp<SM_SPIN>(B_(15), n & 1, abort_flag, p.err, 0x8100u);
      if (!ok) break;
      tcgen05_fence_after();
      const int key0 = j * FA_T + half * 64;
      const int cls = PACKED ? block_class(q0 + (warp & 3) * 32, 32, key0, 64, st_min, st_max)
                             : j == qt ? BLOCK_SOME : BLOCK_ALL;
      uint32_t r[64];
#pragma unroll
      for (int c = 0; c < 4; ++c) tmem_ld16(tS + t_lane + half * 64 + c * 16, r + c * 16);
      tmem_wait_ld();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(8));        // S may be overwritten
      // this half's maximum of the row, then the partner's through its tagged slot
      float mt = -1e30f;
      if (cls == BLOCK_SOME) mt = fwd_max_tile<true>(r, key0, qi, st, mt);
      else if (!PACKED || cls == BLOCK_ALL) mt = fwd_max_tile<false>(r, 0, 0, 0, mt);
      const unsigned long long tag = (unsigned long long)(unsigned)(j + 1) << 32;
      xslot[((j & 1) * 2 + half) * FA_T + qr] = tag | (unsigned long long)__float_as_uint(mt);
      float mo = -1e30f;
      {
        volatile unsigned long long* theirs = xslot + ((j & 1) * 2 + (1 - half)) * FA_T + qr;
        long long t0 = 0;
        for (unsigned spins = 0;; ++spins) {
          const unsigned long long v = *theirs;
          if ((v >> 32) == (unsigned long long)(unsigned)(j + 1)) {
            mo = __uint_as_float((uint32_t)v);
            break;
          }
          if ((spins & 255u) == 255u) {
            if (*abort_flag) { ok = false; break; }
            if (t0 == 0) t0 = clock64();
            else if (clock64() - t0 > WAIT_BUDGET_CYCLES) {
              *abort_flag = 1u;
              if (atomicCAS(p.err, 0u, VKG_ERR_WAIT_TIMEOUT) == 0u) p.err[1] = 0x8150u;
              __threadfence_system();
              ok = false;
              break;
            }
          }
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const float m_row = fmaxf(mt, mo) * p.cscale;
      // the previous P V has retired: the P buffer is free and O~ is quiet
      ok = mbar_wait_warp<SM_SPIN>(B_(10), (n & 1) ^ 1u, abort_flag, p.err, 0x8200u);
      if (!ok) break;
      if (n == 0) {
        m_ref = m_row;
      } else {
        const bool grow = m_row > m_ref + FW1_LAZY;
        if (__any_sync(0xffffffffu, grow)) {
          // rescale this half's 32 columns of O~ (aligned TMEM accesses: the whole warp goes)
          const float alpha = grow ? vkg_ex2(m_ref - m_row) : 1.0f;
          tcgen05_fence_after();
#pragma unroll 1
          for (int c = 0; c < 2; ++c) {          // 16 columns at a time: r[] is still live
            uint32_t o[16];
            tmem_ld16(tO + t_lane + half * 32 + c * 16, o);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * alpha);
            tmem_st16(tO + t_lane + half * 32 + c * 16, o);
          }
          tmem_wait_st();
          l *= alpha;
          if (grow) m_ref = m_row;
        }
      }
      const float nm = -m_ref;
      // P~ packed two keys per register, overwriting the scores they came from, then into
      // this half's 32 columns of the P~ area
      if (cls == BLOCK_SOME) {
        l += fwd_p_pack<true>(r, key0, qi, st, p.cscale, nm);
      } else if (!PACKED || cls == BLOCK_ALL) {
        l += fwd_p_pack<false>(r, 0, 0, 0, p.cscale, nm);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) r[i] = 0u;
      }
      tmem_st16(tP + t_lane + half * 32, r);
      tmem_st16(tP + t_lane + half * 32 + 16, r + 16);
      tmem_wait_st();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(9));        // this warp's part of P~ is in tensor memory
    }
    // row sums of the two halves (both hold the same reference maximum)
    float* xchg = reinterpret_cast<float*>(gbase + FW_XCHG + 2 * 2 * FA_T * 8);
    xchg[half * 128 + qr] = l;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    l = xchg[qr] + xchg[128 + qr];
    const float inv_l = 1.0f / l;               // l > 0: key == query is always valid
    if (half == 0 && q_ok) p.lse2[(size_t)(b * p.H + h) * p.T + qi] = m_ref + log2f(l);
    if (ok) ok = mbar_wait_warp<SM_SPIN>(B_(11), 0, abort_flag, p.err, 0x8300u);
    if (ok) {
      tcgen05_fence_after();
      uint32_t r[32];
      tmem_ld16(tO + t_lane + half * 32, r);
      tmem_ld16(tO + t_lane + half * 32 + 16, r + 16);
      tmem_wait_ld();
      uint4 hv[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        __half2 h2[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          h2[e] = __floats2half2_rn(__uint_as_float(r[u * 8 + 2 * e]) * inv_l,
                                    __uint_as_float(r[u * 8 + 2 * e + 1]) * inv_l);
        hv[u] = *reinterpret_cast<uint4*>(h2);
      }
      const int q_w = q0 + (warp & 3) * 32;
      __half* dst = p.out + (size_t)(row0 + q_w) * p.D + h * FA_HD + half * 32;
      warp_store_rows<4>(hv, gbase + F1_OUT + (warp - 2) * 2048, lane, reinterpret_cast<uint8_t*>(dst),
                         (size_t)p.D * 2, p.T - q_w);
    }
  }

  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, 256);
  }
}

// ---- backward --------------------------------------------------------------------------
//
// Two persistent kernels, one CTA per SM, 24 warps each:
//   warp 0        TMA producer
//   warp 1        S and dP products        warp 2   the gradient products (dQ, or dV and dK)
//   warps 4..7    epilogue: read a finished item's accumulators out, store them, fold their column
//                 sums; in the dQ kernel also delta = rowsum(dO * O) of the item ahead
//   warps 8..23   softmax: four per TMEM lane quarter, 32 of a tile's 128 columns each
// The pipeline runs across items: an item's own operands have two buffers, so the next item's are
// there when its first products are wanted, and nothing the softmax warps do depends on where an
// item ends.  Before (single buffers, accumulators read out and delta formed by the softmax warps) an
// item boundary cost 5000 cycles, 16 to 18 us of each kernel's 50 at 8 x 1024 tokens, 12 heads.
// Registers: 768 threads are launched with 80 each; the softmax warps, which hold 64 scores and
// gradients at a time, take 96 of what the other eight warps give back.  That request is the one wait
// without a limit: with fewer registers at launch it would never be met, so the host compares the split
// with what the kernels were compiled to before it launches them (bwd_registers).
constexpr int BW_EPI_WARP = 4, BW_EPI_WARPS = 4, BW_SM_WARP = 8, BW_SM_WARPS = 16;
constexpr int BW_THREADS = (BW_SM_WARP + BW_SM_WARPS) * 32;
constexpr int BW_REGS_ISSUE = 40, BW_REGS_EPI = 56, BW_REGS_SM = 96;
constexpr int BW_REGS_SPLIT = BW_EPI_WARP * BW_REGS_ISSUE + BW_EPI_WARPS * BW_REGS_EPI + BW_SM_WARPS * BW_REGS_SM;
constexpr int BW_REGS_LAUNCH = BW_REGS_SPLIT / (BW_SM_WARP + BW_SM_WARPS);      // a thread's share
static_assert(BW_REGS_LAUNCH * (BW_SM_WARP + BW_SM_WARPS) == BW_REGS_SPLIT && BW_REGS_LAUNCH == 80,
              "the split is 80 registers a thread, which 768 threads leave room for");

template <int N>
__device__ __forceinline__ void regs_less() {
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_more() {
  asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}

// A warp's 32 rows x 8 NU accumulator columns (lane = row) as fp16 into its staging slice: rows of NU
// 16-byte pieces, piece u of row r at u ^ (r & (NU - 1)).
template <int NU>
__device__ __forceinline__ void stage_acc(uint32_t taddr, uint8_t* stage, int lane) {
#pragma unroll 1
  for (int c = 0; c < NU / 4; ++c) {
    uint32_t rr[32];
    tmem_ld16(taddr + c * 32, rr);
    tmem_ld16(taddr + c * 32 + 16, rr + 16);
    tmem_wait_ld();
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __half2 h = __floats2half2_rn(__uint_as_float(rr[u * 8 + 2 * e]),
                                            __uint_as_float(rr[u * 8 + 2 * e + 1]));
        w[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
      *reinterpret_cast<uint4*>(stage + lane * (NU * 16) + (((c * 4 + u) ^ (lane & (NU - 1))) << 4)) =
          make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

// The staged slice to global rows of `pitch` bytes (32 / NU whole rows per store instruction) and, with
// `sums`, its 8 NU column sums over the rows_ok rows that exist, as stored: NU / 4 adjacent columns per
// lane, the rows in a fixed tree (r + r+16, then 8, 4, 2, 1 apart).
template <int NU>
__device__ __forceinline__ void store_staged(const uint8_t* stage, int lane, uint8_t* dst_row0, size_t pitch,
                                             int rows_ok, float* sums) {
  static_assert(NU == 4 || NU == 8, "32 or 64 columns");
  const int u = lane % NU;
#pragma unroll
  for (int i = 0; i < NU; ++i) {
    const int row = i * (32 / NU) + lane / NU;
    const uint4 x = *reinterpret_cast<const uint4*>(stage + row * (NU * 16) + ((u ^ (row & (NU - 1))) << 4));
    if (row < rows_ok) *reinterpret_cast<uint4*>(dst_row0 + (size_t)row * pitch + u * 16) = x;
  }
  if (!sums) return;
  // NU = 4: a lane's one column is the half of its column pair that its lowest bit names
  const int pair = NU == 8 ? lane : lane >> 1;
  const int piece = pair >> 2, word = (pair & 3) * 4;
  auto at = [&](int r) -> float2 {
    const __half2 h = *reinterpret_cast<const __half2*>(stage + r * (NU * 16) + ((piece ^ (r & (NU - 1))) << 4) + word);
    return r < rows_ok ? __half22float2(h) : make_float2(0.f, 0.f);
  };
  auto add = [](float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); };
  // the tree from its leaves: t8(r) covers rows r, r+16, r+8, r+24
  auto t8 = [&](int r) { return add(add(at(r), at(r + 16)), add(at(r + 8), at(r + 24))); };
  auto t4 = [&](int r) { return add(t8(r), t8(r + 4)); };
  auto t2 = [&](int r) { return add(t4(r), t4(r + 2)); };
  const float2 sum = add(t2(0), t2(1));
  if (NU == 8) {                   // one by one: the caller's scratch need not start on 8 bytes
    sums[2 * lane] = sum.x;
    sums[2 * lane + 1] = sum.y;
  } else {
    sums[lane] = (lane & 1) ? sum.y : sum.x;
  }
}

// Item number j of persistent CTA c out of G: rows of G items are dealt left to right and right
// to left in turn, which spreads items sorted by falling cost almost evenly (within 3 % of the
// mean for 8 query tiles x 96 heads on 148 CTAs; plain round-robin is 16 % off).
__device__ __forceinline__ int snake_item(int j, int G, int c) {
  return j * G + ((j & 1) ? G - 1 - c : c);
}

// dK / dV: an item is a (key tile, head, sequence), heaviest key tile first, and loops over the query
// tiles at or below the diagonal.  The scores are formed transposed, S^T = K Q^T and dP^T = V dO^T
// (TMEM lane = key, column = query), so that P^T and dS^T, which dV += P^T dO and dK += dS^T Q want as
// A operands, go back into tensor memory (fp16 pairs of queries) and never through shared memory:
// writing both there (64 KB a step beside the tensor core's own reads of it) took 670 of a step's
// 2150 cycles.  lse and delta then belong to columns: a warp keeps those of its 32 queries in 256
// bytes of shared memory, read as broadcasts.
// TMEM columns: S^T [0, 128) dP^T [128, 256) dV [256, 320) dK [320, 384) P^T [384, 448) dS^T [448, 512).
constexpr int KV_STAGES = 3;
constexpr int KV_K = 0,                                        // two buffers of K and V
              KV_Q = 4 * FA_TILE_BYTES, KV_DO = (4 + KV_STAGES) * FA_TILE_BYTES,
              KV_OUT = (4 + 2 * KV_STAGES) * FA_TILE_BYTES,    // staging: dV and dK of 32 keys per epilogue warp
              KV_STAT = KV_OUT + BW_EPI_WARPS * 8192,          // (-lse, -delta scale) of 32 queries per softmax warp
              KV_SEG = KV_STAT + BW_SM_WARPS * 256,            // and where their samples start
              KV_TILES = KV_SEG + BW_SM_WARPS * 128,           // packed: the query tiles of each item that count
              KV_BAR = KV_TILES + SEG_ITEMS * 4, KV_SMEM = KV_BAR + 256 + 1024;
static_assert(KV_SMEM <= 227 * 1024, "dK / dV kernel: shared memory");
constexpr int KV_KV_FULL = 0, KV_KV_FREE = 2, KV_SDP_FULL = 4, KV_SDP_FREE = 5, KV_PDS_FULL = 6, KV_PDS_FREE = 7,
              KV_OUT_FULL = 8, KV_ACC_FREE = 10, KV_QD_FULL = 11, KV_QD_EMPTY = 11 + KV_STAGES,
              KV_NBAR = 11 + 2 * KV_STAGES;

// P and dS = P (dP - delta) scale of one key row against 16 queries, as fp16 pairs (queries 2i, 2i + 1)
// in pp[i] and pd[i], ready for tcgen05.st.  P is rebuilt from the saved log-sum-exp; stat holds
// (-lse2, -delta scale) per query, -lse2 = -inf for a query past the end of the sequence, which makes
// its P exactly 0: an element costs two FMAs, one exp2, one multiply and the conversions.  The
// per-element tests, MASK = 1 causal, 2 packed samples too, are only compiled into the tiles that need
// them.
template <int MASK>
__device__ __forceinline__ void bwd_pds_pack(const uint32_t* rs, const uint32_t* rdp, const float4* stat,
                                             const int* seg, int q0, int key, float cscale, float scale,
                                             uint32_t* pp, uint32_t* pd) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float4 s2 = stat[i];
    const int2 sg = MASK == 2 ? reinterpret_cast<const int2*>(seg)[i] : make_int2(0, 0);
    const float nlse[2] = {s2.x, s2.z}, dsc[2] = {s2.y, s2.w};
    float pv[2], dv[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int idx = 2 * i + w;
      float pr = vkg_ex2(fmaf(__uint_as_float(rs[idx]), cscale, nlse[w]));
      if (MASK) {
        bool off = key > q0 + idx;
        if (MASK == 2) off |= key < (w ? sg.y : sg.x);     // not ||, which makes a branch of the load
        if (off) pr = 0.f;
      }
      pv[w] = pr;
      dv[w] = pr * fmaf(__uint_as_float(rdp[idx]), scale, dsc[w]);
    }
    const __half2 hp = __floats2half2_rn(pv[0], pv[1]), hd = __floats2half2_rn(dv[0], dv[1]);
    pp[i] = *reinterpret_cast<const uint32_t*>(&hp);
    pd[i] = *reinterpret_cast<const uint32_t*>(&hd);
  }
}

// Query tile after `it` (counted from the item's first) that counts; ni past the last one.
__device__ __forceinline__ int next_tile(bool skip, uint32_t tiles, int it, int ni) {
  ++it;
  if (!skip || it >= ni) return it;
  const uint32_t left = tiles >> it;
  return left ? it + __ffs((int)left) - 1 : ni;
}

template <bool PACKED>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_kv_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tmdo,
                   const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + KV_BAR;
  auto B_ = [bar](int i) { return bar + 8u * i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + KV_BAR + 192);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(gbase + KV_BAR + 200);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int HB = p.H * p.B;
  const int n_items = p.nqt * HB, G = (int)gridDim.x;

  pdl_trigger();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm);
    prefetch_tensormap(&tmdo);
    for (int i = 0; i < KV_NBAR; ++i)
      mbar_init(B_(i), i == KV_SDP_FREE || i == KV_PDS_FULL ? BW_SM_WARPS : i == KV_ACC_FREE ? BW_EPI_WARPS : 1);
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();
  // packed: bit i of an item's entry says that query tile kt + i has a row whose sample begins before
  // the end of key tile kt; the diagonal tile always counts
  const bool skip = PACKED && p.skip_tiles;
  uint32_t* tiles_s = reinterpret_cast<uint32_t*>(gbase + KV_TILES);
  if (skip) {
    if (threadIdx.x < SEG_ITEMS) tiles_s[threadIdx.x] = 1u;
    __syncthreads();
    // one (item, query tile) per warp and round: 700 cycles each, the wait for the starts
    constexpr int WARPS = BW_THREADS / 32;
    for (int j = 0; j < SEG_ITEMS; ++j) {
      const int item = snake_item(j, G, (int)blockIdx.x);
      if (item >= n_items) break;
      const int kt = item / HB, ni = p.nqt - kt;
      for (int i = 1 + (warp + 5 * j) % WARPS; i < ni; i += WARPS) {
        const int st = tile_first_start(p.seg + ((item % HB) / p.H) * p.T, (kt + i) * FA_T, p.T, lane);
        if (lane == 0 && st < (kt + 1) * FA_T) atomicOr(&tiles_s[j], 1u << i);
      }
    }
    __syncthreads();
  }
  auto item_tiles = [&](int j) { return skip && j < SEG_ITEMS ? tiles_s[j] : ~0u; };
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tdP = tmem + 128, tdV = tmem + 256, tdK = tmem + 320, tP = tmem + 384, tdS = tmem + 448;

  if (warp < BW_EPI_WARP) {
    regs_less<BW_REGS_ISSUE>();
    if (warp == 0) {
      if (lane == 0) {
        int j = 0, s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (;; ++j) {
          const int item = snake_item(j, G, (int)blockIdx.x);
          if (item >= n_items || !ok) break;
          const int kt = item / HB, hb = item % HB;
          const int h = hb % p.H, b = hb / p.H;
          const int row0 = b * p.T, k0 = kt * FA_T, ni = p.nqt - kt;
          const int kb = j & 1;
          // K / V of the item before last are read by its S / dP products only
          if (!mbar_wait<true>(B_(KV_KV_FREE + kb), ((j >> 1) & 1) ^ 1u, abort_flag, p.err, 0x4900u)) break;
          mbar_expect_tx(B_(KV_KV_FULL + kb), 2 * FA_TILE_BYTES);
          tma_load_2d(base + KV_K + (2 * kb) * FA_TILE_BYTES, &tm, B_(KV_KV_FULL + kb), p.D + h * FA_HD, row0 + k0);
          tma_load_2d(base + KV_K + (2 * kb + 1) * FA_TILE_BYTES, &tm, B_(KV_KV_FULL + kb), 2 * p.D + h * FA_HD,
                      row0 + k0);
          const uint32_t tiles = item_tiles(j);
          for (int it = 0; it < ni; it = next_tile(skip, tiles, it, ni)) {
            if (!mbar_wait<true>(B_(KV_QD_EMPTY + s), ph ^ 1u, abort_flag, p.err, 0x4100u + s)) {
              ok = false;
              break;
            }
            mbar_expect_tx(B_(KV_QD_FULL + s), 2 * FA_TILE_BYTES);
            const int qrow = row0 + (kt + it) * FA_T;
            tma_load_2d(base + KV_Q + s * FA_TILE_BYTES, &tm, B_(KV_QD_FULL + s), h * FA_HD, qrow);
            tma_load_2d(base + KV_DO + s * FA_TILE_BYTES, &tmdo, B_(KV_QD_FULL + s), h * FA_HD, qrow);
            if (++s == KV_STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
    } else if (warp == 1) {
      // S^T = K Q^T and dP^T = V dO^T of every step (dV / dK are issued by a warp of their own: one
      // warp's stream of waits, instructions and commits for both paced the step).  The whole warp runs
      // this converged; one elected lane issues each tcgen05 instruction.
      const uint32_t idesc_s = make_idesc(0, 0, 0, FA_T);    // [key x hd] . [q x hd]^T
      const uint32_t d_hi = smem_desc_hi(1024);              // descriptor halves (tcgen05.cuh)
      const uint32_t k_lo = smem_desc_lo(base + KV_K, 16), v_lo = smem_desc_lo(base + KV_K + FA_TILE_BYTES, 16);
      const uint32_t q_lo = smem_desc_lo(base + KV_Q, 16), do_lo = smem_desc_lo(base + KV_DO, 16);
      int s = 0;
      uint32_t ph = 0, par = 0;
      bool ok = true;
      for (int j = 0; ok; ++j) {
        const int item = snake_item(j, G, (int)blockIdx.x);
        if (item >= n_items) break;
        const int ni = p.nqt - item / HB;
        const int kb = j & 1;
        const uint32_t ko = (uint32_t)(2 * kb) * (FA_TILE_BYTES >> 4);
        ok = mbar_wait_warp<true>(B_(KV_KV_FULL + kb), (j >> 1) & 1, abort_flag, p.err, 0x4200u);
        const uint32_t tiles = item_tiles(j);
        for (int it = 0, next; it < ni && ok; it = next) {
          next = next_tile(skip, tiles, it, ni);
          ok = mbar_wait_warp<true>(B_(KV_QD_FULL + s), ph, abort_flag, p.err, 0x4300u + s) &&
               mbar_wait_warp<true>(B_(KV_SDP_FREE), par ^ 1u, abort_flag, p.err, 0x4400u);
          if (!ok) break;
          tcgen05_fence_after();
          const uint32_t so = (uint32_t)s * (FA_TILE_BYTES >> 4);
          umma_f16_chain<4>(tS, k_lo + ko, 2, q_lo + so, 2, d_hi, idesc_s, 0u);
          umma_f16_chain<4>(tdP, v_lo + ko, 2, do_lo + so, 2, d_hi, idesc_s, 0u);
          umma_commit_one(B_(KV_SDP_FULL));
          if (next >= ni) umma_commit_one(B_(KV_KV_FREE + kb));    // the item's K / V may be replaced
          par ^= 1u;
          if (++s == KV_STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    } else if (warp == 2) {
      // dV += P^T dO and dK += dS^T Q of every step.  Its commits cover this warp's instructions
      // only; a Q / dO stage is free when dV / dK of its step have retired, because the S / dP
      // that read it retired before the softmax warps could produce the P / dS these waited for.
      const uint32_t idesc_g = make_idesc(0, 0, 1, FA_HD);   // [key x q] in tensor memory . [q x hd] (MN-major)
      const uint32_t d_hi = smem_desc_hi(1024);
      const uint32_t qm_lo = smem_desc_lo(base + KV_Q, 8192), dom_lo = smem_desc_lo(base + KV_DO, 8192);
      int g = 0, s = 0;
      bool ok = true;
      for (int j = 0; ok; ++j) {
        const int item = snake_item(j, G, (int)blockIdx.x);
        if (item >= n_items) break;
        const int ni = p.nqt - item / HB;
        const uint32_t tiles = item_tiles(j);
        for (int it = 0, next; it < ni; it = next, ++g) {
          next = next_tile(skip, tiles, it, ni);
          ok = mbar_wait_warp<true>(B_(KV_PDS_FULL), g & 1, abort_flag, p.err, 0x4500u);     // P / dS written
          if (!ok) break;
          if (it == 0) {                       // the previous item's dV / dK have been read out
            ok = mbar_wait_warp<true>(B_(KV_ACC_FREE), (j & 1) ^ 1u, abort_flag, p.err, 0x4a00u);
            if (!ok) break;
          }
          tcgen05_fence_after();
          const uint32_t so = (uint32_t)s * (FA_TILE_BYTES >> 4);
          umma_f16_ts_chain<8>(tdV, tP, dom_lo + so, 128, d_hi, idesc_g, it ? 1u : 0u);
          umma_f16_ts_chain<8>(tdK, tdS, qm_lo + so, 128, d_hi, idesc_g, it ? 1u : 0u);
          umma_commit_one(B_(KV_QD_EMPTY + s));   // Q / dO stage free
          umma_commit_one(B_(KV_PDS_FREE));       // P / dS may be overwritten
          if (next >= ni) umma_commit_one(B_(KV_OUT_FULL + (j & 1)));
          if (++s == KV_STAGES) s = 0;
        }
      }
    }
  } else if (warp < BW_SM_WARP) {
    // dV / dK of a finished item: into staging as fp16, accumulators handed back, then stored (slices 2
    // and 1 of dqkv) and added up by columns
    regs_less<BW_REGS_EPI>();
    const int w = warp & 3;
    const uint32_t t_lane = ((uint32_t)(w * 32)) << 16;
    uint8_t* stage = gbase + KV_OUT + w * 8192;
    for (int j = 0;; ++j) {
      const int item = snake_item(j, G, (int)blockIdx.x);
      if (item >= n_items) break;
      if (snake_item(j + 1, G, (int)blockIdx.x) >= n_items) break;   // the last one: see the softmax warps
      const int kt = item / HB, hb = item % HB;
      const int h = hb % p.H, b = hb / p.H;
      if (!mbar_wait_warp<SM_SPIN>(B_(KV_OUT_FULL + (j & 1)), (j >> 1) & 1, abort_flag, p.err, 0x4800u)) break;
      tcgen05_fence_after();
      stage_acc<8>(tdV + t_lane, stage, lane);
      stage_acc<8>(tdK + t_lane, stage + 4096, lane);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(KV_ACC_FREE));     // the accumulators may be overwritten
      const int key_w = kt * FA_T + w * 32;            // first key of this warp's 32 rows
      float* sums = p.colsum ? p.colsum + ((size_t)(b * p.nqt + kt) * 4 + w) * 3 * p.D + h * FA_HD : nullptr;
#pragma unroll 1
      for (int slice = 2; slice >= 1; --slice) {
        __half* dst = p.dqkv + (size_t)(b * p.T + key_w) * 3 * p.D + slice * p.D + h * FA_HD;
        store_staged<8>(stage + (2 - slice) * 4096, lane, reinterpret_cast<uint8_t*>(dst), (size_t)3 * p.D * 2,
                        p.T - key_w, sums ? sums + slice * p.D : nullptr);
      }
      __syncwarp();                                    // the staging is filled again
    }
  } else {
    regs_more<BW_REGS_SM>();
    const int part = (warp - BW_SM_WARP) >> 2;   // which 32 of the tile's 128 queries
    const int r = (warp & 3) * 32 + lane;        // key within the tile = TMEM lane
    const uint32_t t_lane = ((uint32_t)((warp & 3) * 32)) << 16;
    float2* stat = reinterpret_cast<float2*>(gbase + KV_STAT + (warp - BW_SM_WARP) * 256);
    int* seg_s = reinterpret_cast<int*>(gbase + KV_SEG + (warp - BW_SM_WARP) * 128);
    bool ok = true;
    // statistics of the query this lane looks after (part * 32 + lane) in the step ahead, fetched while
    // this one is worked on (a load from global memory at the start of a step would sit on the critical
    // path)
    float lse_n = 0.f, dl_n = 0.f;
    int st_n = 0;
    auto fetch_stat = [&](int hb, int qt) {
      const int qi = qt * FA_T + part * 32 + lane;
      const bool q_ok = qi < p.T;
      const int i = hb * p.T + (q_ok ? qi : 0);
      // a query past the end of the sequence gets lse = +inf, hence P = 0 and dS = 0
      lse_n = q_ok ? p.lse2[i] : INFINITY;
      dl_n = p.delta[i];
      if (PACKED) st_n = q_ok ? (int)p.seg[(hb / p.H) * p.T + qi] : 0;
    };
    if ((int)blockIdx.x < n_items) fetch_stat((int)blockIdx.x % HB, (int)blockIdx.x / HB);
    int g = 0, last = -1, last_j = 0;
    // Barriers are looked at ahead of need, and waited for only if they were not complete by then: a
    // wait that is already satisfied takes 200 to 300 cycles beside a busy tensor core.
    bool ready = false;
    for (int j = 0; ok; ++j) {
      const int item = snake_item(j, G, (int)blockIdx.x);
      if (item >= n_items) break;
      const int kt = item / HB, hb = item % HB;
      const int key = kt * FA_T + r;
      last = item;
      last_j = j;
      const uint32_t tiles = item_tiles(j);
      for (int qt = kt, next; qt < p.nqt && ok; qt = next, ++g) {
        next = kt + next_tile(skip, tiles, qt - kt, p.nqt - kt);
        stat[lane] = make_float2(-lse_n, -dl_n * p.scale);
        int cls = qt == kt ? BLOCK_SOME : BLOCK_ALL;
        if (PACKED) {
          seg_s[lane] = st_n;
          cls = block_class(qt * FA_T + part * 32, 32, key - lane, 32, __reduce_min_sync(0xffffffffu, st_n),
                            __reduce_max_sync(0xffffffffu, st_n));
        }
        __syncwarp();
        if (next < p.nqt) {
          fetch_stat(hb, next);
        } else {
          const int nxt = snake_item(j + 1, G, (int)blockIdx.x);
          if (nxt < n_items) fetch_stat(nxt % HB, nxt / HB);
        }
        ok = ready || mbar_wait_warp<SM_SPIN>(B_(KV_SDP_FULL), g & 1, abort_flag, p.err, 0x4600u);
        if (!ok) break;
        tcgen05_fence_after();
        uint32_t rs[32], rdp[32];
        tmem_ld16(tS + t_lane + part * 32, rs);
        tmem_ld16(tS + t_lane + part * 32 + 16, rs + 16);
        tmem_ld16(tdP + t_lane + part * 32, rdp);
        tmem_ld16(tdP + t_lane + part * 32 + 16, rdp + 16);
        tmem_wait_ld();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(B_(KV_SDP_FREE));          // S / dP may be overwritten
        // P and dS, overwriting the scores and products they came from
        const float4* st4 = reinterpret_cast<const float4*>(stat);
        const int q0 = qt * FA_T + part * 32;
        if (cls == BLOCK_SOME) bwd_pds_pack<PACKED ? 2 : 1>(rs, rdp, st4, seg_s, q0, key, p.cscale, p.scale, rs, rdp);
        else if (!PACKED || cls == BLOCK_ALL) bwd_pds_pack<0>(rs, rdp, st4, nullptr, 0, 0, p.cscale, p.scale, rs, rdp);
        ready = mbar_test_wait(B_(KV_PDS_FREE), (g & 1) ^ 1u) != 0;
        if (cls == BLOCK_SOME) {
          bwd_pds_pack<PACKED ? 2 : 1>(rs + 16, rdp + 16, st4 + 8, seg_s + 16, q0 + 16, key, p.cscale, p.scale, rs + 8,
                                       rdp + 8);
        } else if (!PACKED || cls == BLOCK_ALL) {
          bwd_pds_pack<0>(rs + 16, rdp + 16, st4 + 8, nullptr, 0, 0, p.cscale, p.scale, rs + 8, rdp + 8);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) rs[i] = rdp[i] = 0u;
        }
        // dV / dK of step g - 1 done
        ok = __all_sync(0xffffffffu, ready) ||
             mbar_wait_warp<SM_SPIN>(B_(KV_PDS_FREE), (g & 1) ^ 1u, abort_flag, p.err, 0x4700u);
        if (!ok) break;
        tcgen05_fence_after();
        tmem_st16(tP + t_lane + part * 16, rs);
        tmem_st16(tdS + t_lane + part * 16, rdp);
        ready = mbar_test_wait(B_(KV_SDP_FULL), (g & 1) ^ 1u) != 0;
        tmem_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(B_(KV_PDS_FULL));
        ready = __all_sync(0xffffffffu, ready);
      }
    }
    // The CTA's last item (its only one in a small problem) has nothing to overlap with: all sixteen
    // warps read it out, 32 columns each (dV by parts 0 and 1, dK by 2 and 3), through the idle ring.
    // They have waited for no other item's KV_OUT_FULL, and a parity wait also passes while its barrier is
    // a phase behind.  Hence a barrier for even items and one for odd ones: a phase behind is then item
    // last_j - 2, whose barrier has completed.  The last wait for KV_PDS_FREE was for a step of the last
    // item or of the one before it (every item has a step), the products of either came after those of
    // item last_j - 1's first step, and these after KV_ACC_FREE of item last_j - 2, which its readers signal
    // only once they have seen its KV_OUT_FULL.  With one barrier, a last item of one step could find the
    // phase of item last_j - 1 still open: its KV_PDS_FREE and KV_OUT_FULL are two commits.
    if (ok && last >= 0 &&
        mbar_wait_warp<SM_SPIN>(B_(KV_OUT_FULL + (last_j & 1)), (last_j >> 1) & 1, abort_flag, p.err, 0x4c00u)) {
      tcgen05_fence_after();
      uint8_t* stage = gbase + KV_Q + (warp - BW_SM_WARP) * 2048;
      stage_acc<4>(tdV + t_lane + part * 32, stage, lane);
      __syncwarp();
      const int kt = last / HB, hb = last % HB, b = hb / p.H;
      const int key_w = kt * FA_T + (warp & 3) * 32;
      const int col = (part < 2 ? 2 : 1) * p.D + (hb % p.H) * FA_HD + (part & 1) * 32;
      store_staged<4>(stage, lane, reinterpret_cast<uint8_t*>(p.dqkv + (size_t)(b * p.T + key_w) * 3 * p.D + col),
                      (size_t)3 * p.D * 2, p.T - key_w,
                      p.colsum ? p.colsum + ((size_t)(b * p.nqt + kt) * 4 + (warp & 3)) * 3 * p.D + col : nullptr);
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// dQ: an item is a (query tile, head, sequence), heaviest query tile first, and loops over the key
// tiles up to the diagonal.  Q / dO / O are the per-item operands, K / V the per-step ones, in a ring
// of three stages: a stage is read by S / dP of its step and again by dQ of the same step a softmax
// later.
// dS never passes through shared memory: the softmax warps write it (fp16 pairs) into one of
// two areas of tensor memory with tcgen05.st, and dQ += dS K reads it there as the A operand.
// The warps that issue the MMAs keep their loops as short as they can be (one elected lane per
// instruction, descriptor halves stepped by adds, no wait that another wait implies): a wait that is
// already satisfied costs such a warp about 180 cycles and a loop iteration 400.  Splitting a step into
// two half-steps with two softmax groups half a step apart doubled their waits and commits and
// measured 15 % slower, although the softmax warps then idled less.
// This kernel also forms delta = rowsum(dO * O) (tkernels.py:176-179 computes the same number
// as sum_j dP_ij P_ij): the epilogue warps add a row's 64 products up from the O and dO tiles of the
// item ahead, for the softmax warps and, written out, for the dK / dV kernel, which is launched after
// this one.
// TMEM columns: S [0, 128) dP [128, 256) dQ [256 + 64 a, +64) of two items in turn, dS [384 + 64 b, +64).
constexpr int DQ_STAGES = 3;
constexpr int DQ_Q = 0,                                        // two buffers of Q, dO and O
              DQ_K = 6 * FA_TILE_BYTES, DQ_V = (6 + DQ_STAGES) * FA_TILE_BYTES,
              DQ_OUT = (6 + 2 * DQ_STAGES) * FA_TILE_BYTES,    // output staging, one tile
              DQ_DELTA = DQ_OUT + FA_TILE_BYTES,               // [2][128] floats
              DQ_FIRST = DQ_DELTA + 1024,                      // packed: the first key tile of each item that counts
              DQ_BAR = DQ_FIRST + SEG_ITEMS * 4, DQ_SMEM = DQ_BAR + 256 + 1024;
static_assert(DQ_SMEM <= 227 * 1024, "dQ kernel: shared memory");
constexpr int DQ_QD_FULL = 0, DQ_QD_FREE = 2, DQ_OD_FREE = 4, DQ_DL_FULL = 6, DQ_SDP_FULL = 8, DQ_SDP_FREE = 9,
              DQ_DS_FULL = 10, DQ_DS_FREE = 12, DQ_OUT_FULL = 14, DQ_ACC_FREE = 16, DQ_KV_FULL = 18,
              DQ_KV_EMPTY = 18 + DQ_STAGES, DQ_NBAR = 18 + 2 * DQ_STAGES;

// dS = P (dP - delta) scale for 16 keys of one query row, as fp16 pairs (keys 2i, 2i + 1) in
// pk[i], ready for tcgen05.st; P is rebuilt from the saved log-sum-exp as in bwd_pds_pack.
template <bool MASK>
__device__ __forceinline__ void bwd_ds_pack(const uint32_t* rs, const uint32_t* rdp, int key0, int qi,
                                            int st, float cscale, float scale, float nlse, float dsc,
                                            uint32_t* pk) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float dv[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int idx = 2 * i + w;
      float pr = vkg_ex2(fmaf(__uint_as_float(rs[idx]), cscale, nlse));
      if (MASK) {
        const int key = key0 + idx;
        if (key > qi || key < st) pr = 0.f;
      }
      dv[w] = pr * fmaf(__uint_as_float(rdp[idx]), scale, dsc);
    }
    const __half2 h = __floats2half2_rn(dv[0], dv[1]);
    pk[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
}

template <bool PACKED>
__global__ void __launch_bounds__(BW_THREADS, 1)
attn_bwd_q_kernel(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tmdo,
                  const __grid_constant__ CUtensorMap tmo, const AttnParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar = base + DQ_BAR;
  auto B_ = [bar](int i) { return bar + 8u * i; };
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + DQ_BAR + 192);
  volatile uint32_t* abort_flag = reinterpret_cast<volatile uint32_t*>(gbase + DQ_BAR + 200);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int HB = p.H * p.B;
  const int n_items = p.nqt * HB, G = (int)gridDim.x;

  pdl_trigger();
  if (threadIdx.x == 0) {
    prefetch_tensormap(&tm);
    prefetch_tensormap(&tmdo);
    prefetch_tensormap(&tmo);
    for (int i = 0; i < DQ_NBAR; ++i) {
      const bool sm = i == DQ_SDP_FREE || (i >= DQ_DS_FULL && i < DQ_DS_FULL + 2);
      const bool epi = (i >= DQ_OD_FREE && i < DQ_DL_FULL + 2) || (i >= DQ_ACC_FREE && i < DQ_ACC_FREE + 2);
      mbar_init(B_(i), sm ? BW_SM_WARPS : epi ? BW_EPI_WARPS : 1);
    }
    *abort_flag = 0u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  pdl_wait();
  int* first_s = reinterpret_cast<int*>(gbase + DQ_FIRST);
  if (PACKED && p.skip_tiles) {
    for (int j = warp; j < SEG_ITEMS; j += BW_THREADS / 32) {
      const int item = snake_item(j, G, (int)blockIdx.x);
      if (item >= n_items) break;
      const int qt = p.nqt - 1 - item / HB;
      const int st = tile_first_start(p.seg + ((item % HB) / p.H) * p.T, qt * FA_T, p.T, lane);
      if (lane == 0) first_s[j] = min(st / FA_T, qt);
    }
    __syncthreads();
  }
  auto item_first = [&](int j) { return PACKED && p.skip_tiles && j < SEG_ITEMS ? first_s[j] : 0; };
  const uint32_t tmem = *tmem_slot;
  const uint32_t tS = tmem, tdP = tmem + 128, tdQ = tmem + 256, tdS = tmem + 384;

  if (warp < BW_EPI_WARP) {
    regs_less<BW_REGS_ISSUE>();
    if (warp == 0) {
      if (lane == 0) {
        int j = 0, s = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (;; ++j) {
          const int item = snake_item(j, G, (int)blockIdx.x);
          if (item >= n_items || !ok) break;
          const int qt = p.nqt - 1 - item / HB, hb = item % HB;
          const int h = hb % p.H, b = hb / p.H;
          const int row0 = b * p.T, q0 = qt * FA_T, nj = qt + 1;
          const int qb = j & 1;
          const uint32_t qd = base + DQ_Q + (uint32_t)(3 * qb) * FA_TILE_BYTES;
          const uint32_t old = ((j >> 1) & 1) ^ 1u;
          // Q / dO of the item before last have been read by its S / dP, its dO / O by the epilogue warps
          if (!(mbar_wait<true>(B_(DQ_QD_FREE + qb), old, abort_flag, p.err, 0x5900u) &&
                mbar_wait<true>(B_(DQ_OD_FREE + qb), old, abort_flag, p.err, 0x5b00u)))
            break;
          mbar_expect_tx(B_(DQ_QD_FULL + qb), 3 * FA_TILE_BYTES);
          tma_load_2d(qd, &tm, B_(DQ_QD_FULL + qb), h * FA_HD, row0 + q0);
          tma_load_2d(qd + FA_TILE_BYTES, &tmdo, B_(DQ_QD_FULL + qb), h * FA_HD, row0 + q0);
          tma_load_2d(qd + 2 * FA_TILE_BYTES, &tmo, B_(DQ_QD_FULL + qb), h * FA_HD, row0 + q0);
          for (int kt = item_first(j); kt < nj; ++kt) {
            if (!mbar_wait<true>(B_(DQ_KV_EMPTY + s), ph ^ 1u, abort_flag, p.err, 0x5100u + s)) {
              ok = false;
              break;
            }
            mbar_expect_tx(B_(DQ_KV_FULL + s), 2 * FA_TILE_BYTES);
            tma_load_2d(base + DQ_K + s * FA_TILE_BYTES, &tm, B_(DQ_KV_FULL + s), p.D + h * FA_HD, row0 + kt * FA_T);
            tma_load_2d(base + DQ_V + s * FA_TILE_BYTES, &tm, B_(DQ_KV_FULL + s), 2 * p.D + h * FA_HD,
                        row0 + kt * FA_T);
            if (++s == DQ_STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
    } else if (warp == 1) {
      // S = Q K^T and dP = dO V^T of every step.  The whole warp runs this converged; one elected
      // lane issues each tcgen05 instruction.
      const uint32_t idesc_s = make_idesc(0, 0, 0, FA_T);
      const uint32_t d_hi = smem_desc_hi(1024);      // descriptor halves (tcgen05.cuh)
      const uint32_t q_lo = smem_desc_lo(base + DQ_Q, 16), do_lo = smem_desc_lo(base + DQ_Q + FA_TILE_BYTES, 16);
      const uint32_t k_lo = smem_desc_lo(base + DQ_K, 16), v_lo = smem_desc_lo(base + DQ_V, 16);
      int s = 0;
      uint32_t ph = 0, par = 0;
      bool ok = true;
      for (int j = 0; ok; ++j) {
        const int item = snake_item(j, G, (int)blockIdx.x);
        if (item >= n_items) break;
        const int nj = p.nqt - item / HB;               // key tiles of the item: qt + 1
        const int qb = j & 1;
        const uint32_t qo = (uint32_t)(3 * qb) * (FA_TILE_BYTES >> 4);
        ok = mbar_wait_warp<true>(B_(DQ_QD_FULL + qb), (j >> 1) & 1, abort_flag, p.err, 0x5200u);
        for (int kt = item_first(j); kt < nj && ok; ++kt) {
          ok = mbar_wait_warp<true>(B_(DQ_KV_FULL + s), ph, abort_flag, p.err, 0x5300u + s) &&
               mbar_wait_warp<true>(B_(DQ_SDP_FREE), par ^ 1u, abort_flag, p.err, 0x5400u);
          if (!ok) break;
          tcgen05_fence_after();
          const uint32_t so = (uint32_t)s * (FA_TILE_BYTES >> 4);
          umma_f16_chain<4>(tS, q_lo + qo, 2, k_lo + so, 2, d_hi, idesc_s, 0u);
          umma_f16_chain<4>(tdP, do_lo + qo, 2, v_lo + so, 2, d_hi, idesc_s, 0u);
          umma_commit_one(B_(DQ_SDP_FULL));
          if (kt == nj - 1) umma_commit_one(B_(DQ_QD_FREE + qb));    // the item's Q / dO may be replaced
          par ^= 1u;
          if (++s == DQ_STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
    } else if (warp == 2) {
      // dQ += dS K of every step, issued by a warp of its own: the instruction stream of one warp
      // for both (waits, 16 instructions, commits, about 1900 cycles per step next to busy softmax
      // warps) was what paced the kernel.  Its commits cover this warp's instructions only; a
      // K / V stage is free when dQ of its step has retired, because the S / dP that read it
      // retired before the softmax warps could produce the dS this dQ waited for.
      const uint32_t idesc_q = make_idesc(0, 0, 1, FA_HD);   // dS (tensor memory) . K (MN-major), N = 64
      const uint32_t d_hi = smem_desc_hi(1024);
      const uint32_t km_lo = smem_desc_lo(base + DQ_K, 8192);
      int g = 0, s = 0;
      bool ok = true;
      for (int j = 0; ok; ++j) {
        const int item = snake_item(j, G, (int)blockIdx.x);
        if (item >= n_items) break;
        const int nj = p.nqt - item / HB;
        const int ab = j & 1;
        const int first = item_first(j);
        for (int kt = first; kt < nj; ++kt, ++g) {
          const int pb = g & 1;
          ok = mbar_wait_warp<true>(B_(DQ_DS_FULL + pb), (g >> 1) & 1, abort_flag, p.err, 0x5500u);
          if (!ok) break;
          if (kt == first) {                    // dQ of the item before last has been read out
            ok = mbar_wait_warp<true>(B_(DQ_ACC_FREE + ab), ((j >> 1) & 1) ^ 1u, abort_flag, p.err, 0x5a00u);
            if (!ok) break;
          }
          tcgen05_fence_after();
          // K = 128 keys: dS from tensor memory (8 columns per step), K MN-major
          umma_f16_ts_chain<8>(tdQ + 64 * ab, tdS + 64 * pb, km_lo + (uint32_t)s * (FA_TILE_BYTES >> 4), 128, d_hi,
                               idesc_q, kt != first ? 1u : 0u);
          umma_commit_one(B_(DQ_KV_EMPTY + s));   // K / V stage free
          umma_commit_one(B_(DQ_DS_FREE + pb));   // this dS area free
          if (kt == nj - 1) umma_commit_one(B_(DQ_OUT_FULL + ab));
          if (++s == DQ_STAGES) s = 0;
        }
      }
    }
  } else if (warp < BW_SM_WARP) {
    regs_less<BW_REGS_EPI>();
    const int w = warp & 3;
    const int r = w * 32 + lane;                 // query row within the tile = TMEM lane
    uint8_t* stage = gbase + DQ_OUT + w * 4096;
    float* delta_s = reinterpret_cast<float*>(gbase + DQ_DELTA);
    // delta of item j's rows from its dO and O tiles (128-byte rows, 16-byte pieces XOR-ed with the
    // row's low three bits, as the tensor map wrote them).  Item j - 2's delta has been read by then:
    // its dQ, which this warp has stored, came after.
    auto form_delta = [&](int j) -> bool {
      const int item = snake_item(j, G, (int)blockIdx.x);
      const int qb = j & 1;
      if (!mbar_wait_warp<SM_SPIN>(B_(DQ_QD_FULL + qb), (j >> 1) & 1, abort_flag, p.err, 0x5c00u)) return false;
      const uint8_t* dor = gbase + DQ_Q + (3 * qb + 1) * FA_TILE_BYTES + r * 128;
      const uint8_t* orow = dor + FA_TILE_BYTES;
      float dl = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const uint32_t off = ((uint32_t)c ^ (uint32_t)(r & 7)) << 4;
        const uint4 a = *reinterpret_cast<const uint4*>(dor + off);
        const uint4 o = *reinterpret_cast<const uint4*>(orow + off);
        const __half2* ah = reinterpret_cast<const __half2*>(&a);
        const __half2* oh = reinterpret_cast<const __half2*>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 x = __half22float2(ah[e]), y = __half22float2(oh[e]);
          dl = fmaf(x.x, y.x, dl);
          dl = fmaf(x.y, y.y, dl);
        }
      }
      delta_s[qb * FA_T + r] = dl;
      const int qi = (p.nqt - 1 - item / HB) * FA_T + r;
      if (qi < p.T) p.delta_out[(size_t)(item % HB) * p.T + qi] = dl;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(B_(DQ_DL_FULL + qb));
        mbar_arrive(B_(DQ_OD_FREE + qb));
      }
      return true;
    };
    bool ok = (int)blockIdx.x < n_items && form_delta(0);
    for (int j = 0; ok; ++j) {
      const int item = snake_item(j, G, (int)blockIdx.x);
      if (item >= n_items) break;
      if (snake_item(j + 1, G, (int)blockIdx.x) >= n_items) break;   // the last one: see the softmax warps
      ok = form_delta(j + 1);
      if (!ok) break;
      const int qt = p.nqt - 1 - item / HB, hb = item % HB;
      const int h = hb % p.H, b = hb / p.H;
      const int ab = j & 1;
      if (!mbar_wait_warp<SM_SPIN>(B_(DQ_OUT_FULL + ab), (j >> 1) & 1, abort_flag, p.err, 0x5800u)) break;
      tcgen05_fence_after();
      stage_acc<8>(tdQ + 64 * ab + (((uint32_t)(w * 32)) << 16), stage, lane);
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(B_(DQ_ACC_FREE + ab));     // dQ may be overwritten
      const int q_w = qt * FA_T + w * 32;                   // first query row of this warp's 32
      __half* dst = p.dqkv + (size_t)(b * p.T + q_w) * 3 * p.D + h * FA_HD;
      store_staged<8>(stage, lane, reinterpret_cast<uint8_t*>(dst), (size_t)3 * p.D * 2, p.T - q_w,
                      p.colsum ? p.colsum + ((size_t)(b * p.nqt + qt) * 4 + w) * 3 * p.D + h * FA_HD : nullptr);
      __syncwarp();                                         // the staging is filled again
    }
  } else {
    regs_more<BW_REGS_SM>();
    const int part = (warp - BW_SM_WARP) >> 2;   // which 32 of a key tile's 128 keys
    const int r = (warp & 3) * 32 + lane;
    const uint32_t t_lane = ((uint32_t)((warp & 3) * 32)) << 16;
    const float* delta_s = reinterpret_cast<const float*>(gbase + DQ_DELTA);
    bool ok = true;
    // statistics of this thread's query row in an item, fetched one item ahead
    auto item_stat = [&](int item, float& lse, int& st) {
      const int qt = p.nqt - 1 - item / HB, hb = item % HB;
      const int qi = qt * FA_T + r;
      const bool q_ok = qi < p.T;
      lse = p.lse2[(size_t)hb * p.T + (q_ok ? qi : 0)];
      st = (PACKED && q_ok) ? (int)p.seg[(hb / p.H) * p.T + qi] : 0;
    };
    float lse_f = 0.f;
    int st_f = 0;
    if ((int)blockIdx.x < n_items) item_stat((int)blockIdx.x, lse_f, st_f);
    int g = 0, j = 0, last = -1;
    bool ready = false;          // as in the dK / dV kernel
    for (;; ++j) {
      const int item = snake_item(j, G, (int)blockIdx.x);
      if (item >= n_items || !ok) break;
      const int qt = p.nqt - 1 - item / HB, nj = qt + 1;
      const int qi = qt * FA_T + r;
      last = item;
      // a row past the end of the sequence gets lse = +inf, hence P = 0 and dS = 0
      const float nlse = qi < p.T ? -lse_f : -INFINITY;
      const int st = st_f;
      const int st_min = PACKED ? __reduce_min_sync(0xffffffffu, st) : 0;
      const int st_max = PACKED ? __reduce_max_sync(0xffffffffu, st) : 0;
      {
        const int nxt = snake_item(j + 1, G, (int)blockIdx.x);
        if (nxt < n_items) item_stat(nxt, lse_f, st_f);
      }
      ok = mbar_wait_warp<SM_SPIN>(B_(DQ_DL_FULL + (j & 1)), (j >> 1) & 1, abort_flag, p.err, 0x5d00u);
      if (!ok) break;
      const float dsc = -delta_s[(j & 1) * FA_T + r] * p.scale;
      for (int kt = item_first(j); kt < nj && ok; ++kt, ++g) {
        ok = ready || mbar_wait_warp<SM_SPIN>(B_(DQ_SDP_FULL), g & 1, abort_flag, p.err, 0x5600u);
        if (!ok) break;
        tcgen05_fence_after();
        uint32_t rs[32], rdp[32];
        tmem_ld16(tS + t_lane + part * 32, rs);
        tmem_ld16(tS + t_lane + part * 32 + 16, rs + 16);
        tmem_ld16(tdP + t_lane + part * 32, rdp);
        tmem_ld16(tdP + t_lane + part * 32 + 16, rdp + 16);
        tmem_wait_ld();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(B_(DQ_SDP_FREE));
        // dS as fp16 pairs, overwriting the scores they came from
        const int key0 = kt * FA_T + part * 32;
        const int cls = PACKED ? block_class(qi - lane, 32, key0, 32, st_min, st_max)
                               : kt == qt ? BLOCK_SOME : BLOCK_ALL;
        if (cls == BLOCK_SOME) bwd_ds_pack<true>(rs, rdp, key0, qi, st, p.cscale, p.scale, nlse, dsc, rs);
        else if (!PACKED || cls == BLOCK_ALL) bwd_ds_pack<false>(rs, rdp, 0, 0, 0, p.cscale, p.scale, nlse, dsc, rs);
        const int pb = g & 1;
        ready = mbar_test_wait(B_(DQ_DS_FREE + pb), ((g >> 1) & 1) ^ 1u) != 0;
        if (cls == BLOCK_SOME) {
          bwd_ds_pack<true>(rs + 16, rdp + 16, key0 + 16, qi, st, p.cscale, p.scale, nlse, dsc, rs + 8);
        } else if (!PACKED || cls == BLOCK_ALL) {
          bwd_ds_pack<false>(rs + 16, rdp + 16, 0, 0, 0, p.cscale, p.scale, nlse, dsc, rs + 8);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i) rs[i] = 0u;
        }
        // dQ of step g - 2 has read this dS area
        ok = __all_sync(0xffffffffu, ready) ||
             mbar_wait_warp<SM_SPIN>(B_(DQ_DS_FREE + pb), ((g >> 1) & 1) ^ 1u, abort_flag, p.err, 0x5700u);
        if (!ok) break;
        tcgen05_fence_after();
        tmem_st16(tdS + 64 * pb + t_lane + part * 16, rs);
        ready = mbar_test_wait(B_(DQ_SDP_FULL), (g & 1) ^ 1u) != 0;
        tmem_wait_st();
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(B_(DQ_DS_FULL + pb));
        ready = __all_sync(0xffffffffu, ready);
      }
    }
    // the CTA's last item, as in the dK / dV kernel: 32 columns each by parts 0 and 1
    const int la = (j - 1) & 1;
    if (ok && last >= 0 && part < 2 &&
        mbar_wait_warp<SM_SPIN>(B_(DQ_OUT_FULL + la), ((j - 1) >> 1) & 1, abort_flag, p.err, 0x5f00u)) {
      tcgen05_fence_after();
      uint8_t* stage = gbase + DQ_K + (warp - BW_SM_WARP) * 2048;
      stage_acc<4>(tdQ + 64 * la + t_lane + part * 32, stage, lane);
      __syncwarp();
      const int qt = p.nqt - 1 - last / HB, hb = last % HB, b = hb / p.H;
      const int q_w = qt * FA_T + (warp & 3) * 32;
      const int col = (hb % p.H) * FA_HD + part * 32;
      store_staged<4>(stage, lane, reinterpret_cast<uint8_t*>(p.dqkv + (size_t)(b * p.T + q_w) * 3 * p.D + col),
                      (size_t)3 * p.D * 2, p.T - q_w,
                      p.colsum ? p.colsum + ((size_t)(b * p.nqt + qt) * 4 + (warp & 3)) * 3 * p.D + col : nullptr);
    }
  }
  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    long long t0 = clock64();
    while (clock64() - t0 < 2000000ll) {
    }
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// 2-D map over a row-major fp16 matrix (rows x cols), 64-column x 128-row boxes.
int make_map_2d(vkg_device* dev, CUtensorMap* map, const void* ptr, int64_t cols, int64_t rows,
                const char* what) {
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)(cols * 2)};
  cuuint32_t box[2] = {FA_HD, FA_T};
  cuuint32_t estr[2] = {1, 1};
  if (((uintptr_t)ptr & 15) || ((cols * 2) & 15)) {
    vkg_set_error("attention operand %s must be 16-byte aligned with a 16-byte row pitch", what);
    return 1;
  }
  CUresult r = ((EncodeTiledFn)dev->encode_tiled)(
      map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    vkg_set_error("cuTensorMapEncodeTiled failed for %s with code %d", what, (int)r);
    return 1;
  }
  return 0;
}

// Refuses a backward kernel that was compiled to fewer registers a thread than its warps share out.
int bwd_registers(int per_thread) {
  VKG_REQUIRE(per_thread >= BW_REGS_LAUNCH,
              "attn_bwd: the kernels are launched with %d registers a thread, their warps' shares need %d",
              per_thread, BW_REGS_LAUNCH);
  return 0;
}

template <typename Kernel>
int bwd_prepare(Kernel fn, int smem) {
  cudaFuncAttributes attr;
  VKG_CUDA(cudaFuncGetAttributes(&attr, fn));
  if (bwd_registers(attr.numRegs)) return 1;
  VKG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  return 0;
}

}  // namespace

extern "C" int vkg_selftest_attn_registers(int per_thread) { return bwd_registers(per_thread); }

extern "C" int vkg_attn_fwd(vkg_device* dev, const void* qkv16, const uint32_t* seg, void* out16,
                            float* lse2, int B, int T, int H, int hd, float scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(qkv16 && out16 && lse2 && B > 0 && T > 0 && H > 0, "attn_fwd: bad arguments");
  VKG_REQUIRE(hd == FA_HD, "attn_fwd: head dimension must be %d (got %d)", FA_HD, hd);
  VKG_REQUIRE(((uintptr_t)out16 & 15) == 0, "attn_fwd: output must be 16-byte aligned");
  const int D = H * hd;
  CUtensorMap tm;
  if (make_map_2d(dev, &tm, qkv16, 3 * (int64_t)D, (int64_t)B * T, "qkv")) return 1;
  AttnParams p;
  memset(&p, 0, sizeof(p));
  p.B = B; p.T = T; p.H = H; p.D = D;
  p.nqt = (T + FA_T - 1) / FA_T;
  p.scale = scale;
  p.cscale = scale * LOG2E;
  p.seg = seg;
  p.skip_tiles = skip_tiles(seg, p.nqt);
  p.out = (__half*)out16;
  p.lse2 = lse2;
  p.err = dev->err_dev;
  if (!dev->attn_fwd_attr_set) {
    VKG_CUDA(cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  FW_SMEM));
    for (auto fn : {attn_fwd1_kernel<false>, attn_fwd1_kernel<true>})
      VKG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, FW_SMEM));
    dev->attn_fwd_attr_set = true;
  }
  const long long ctas = (long long)p.nqt * H * B;
  VKG_REQUIRE(ctas < (1ll << 31), "attn_fwd: too many tiles");
  VKG_CUDA(vkg_launch(dev, VKG_K_ATTN_FWD | vkg_short_if(ctas <= 2ll * dev->sm_count),
                      !dev->attn_one_pass ? attn_fwd_kernel : seg ? attn_fwd1_kernel<true> : attn_fwd1_kernel<false>,
                      dim3((unsigned)ctas), dim3(FA_THREADS), FW_SMEM, 1, tm, p));
  return vkg_check_launch("attn_fwd_kernel");
}

extern "C" int vkg_attn_bwd(vkg_device* dev, const void* qkv16, const void* dout16, const void* out16,
                            const float* lse2, const uint32_t* seg, void* dqkv16, float* delta,
                            float* dbias, float* dbias_scratch, int B, int T, int H, int hd,
                            float scale) {
  if (vkg_bind(dev)) return 1;
  VKG_REQUIRE(qkv16 && dout16 && out16 && lse2 && dqkv16 && delta && B > 0 && T > 0 && H > 0,
              "attn_bwd: bad arguments");
  VKG_REQUIRE(hd == FA_HD, "attn_bwd: head dimension must be %d (got %d)", FA_HD, hd);
  VKG_REQUIRE(((uintptr_t)dqkv16 & 15) == 0, "attn_bwd: dqkv must be 16-byte aligned");
  const int D = H * hd;
  CUtensorMap tm, tmdo, tmo;
  if (make_map_2d(dev, &tm, qkv16, 3 * (int64_t)D, (int64_t)B * T, "qkv")) return 1;
  if (make_map_2d(dev, &tmdo, dout16, (int64_t)D, (int64_t)B * T, "dO")) return 1;
  if (make_map_2d(dev, &tmo, out16, (int64_t)D, (int64_t)B * T, "O")) return 1;
  AttnParams p;
  memset(&p, 0, sizeof(p));
  p.B = B; p.T = T; p.H = H; p.D = D;
  p.nqt = (T + FA_T - 1) / FA_T;
  p.scale = scale;
  p.cscale = scale * LOG2E;
  p.seg = seg;
  p.skip_tiles = skip_tiles(seg, p.nqt);
  p.lse2 = const_cast<float*>(lse2);
  p.delta = delta;
  p.delta_out = delta;
  p.dqkv = (__half*)dqkv16;
  p.err = dev->err_dev;
  VKG_REQUIRE(!dbias || dbias_scratch, "attn_bwd: dbias needs dbias_scratch");
  p.colsum = dbias ? dbias_scratch : nullptr;
  if (!dev->attn_bwd_attr_set) {
    for (auto fn : {attn_bwd_kv_kernel<false>, attn_bwd_kv_kernel<true>})
      if (bwd_prepare(fn, KV_SMEM)) return 1;
    for (auto fn : {attn_bwd_q_kernel<false>, attn_bwd_q_kernel<true>})
      if (bwd_prepare(fn, DQ_SMEM)) return 1;
    dev->attn_bwd_attr_set = true;
  }
  VKG_REQUIRE((((uintptr_t)dout16 | (uintptr_t)out16) & 15) == 0, "attn_bwd: dO and O must be 16-byte aligned");
  const long long n_items = (long long)p.nqt * H * B;
  VKG_REQUIRE(n_items < (1ll << 31), "attn_bwd: too many tiles");
  // persistent kernels: one CTA per SM (their shared memory allows no more), items dealt in
  // snake order; the dQ kernel goes first because it also writes delta
  const int sms = vkg_persistent_ctas(dev);
  const unsigned ctas = (unsigned)(n_items < sms ? n_items : sms);
  const unsigned family = VKG_K_ATTN_BWD | vkg_short_if(n_items <= sms);
  VKG_CUDA(vkg_launch(dev, family, seg ? attn_bwd_q_kernel<true> : attn_bwd_q_kernel<false>, dim3(ctas),
                      dim3(BW_THREADS), DQ_SMEM, 1, tm, tmdo, tmo, p));
  if (vkg_check_launch("attn_bwd_q_kernel")) return 1;
  VKG_CUDA(vkg_launch(dev, family, seg ? attn_bwd_kv_kernel<true> : attn_bwd_kv_kernel<false>, dim3(ctas),
                      dim3(BW_THREADS), KV_SMEM, 1, tm, tmdo, p));
  if (vkg_check_launch("attn_bwd_kv_kernel")) return 1;
  if (dbias)
    return vkg_launch_col_sum_final(dev, dbias_scratch, dbias, 3 * D, B * p.nqt * 4, 0);
  return 0;
}

extern "C" int64_t vkg_attn_bwd_dbias_scratch_floats(int B, int T, int H, int hd) {
  if (B <= 0 || T <= 0 || H <= 0 || hd <= 0) return 0;
  return (int64_t)B * ((T + FA_T - 1) / FA_T) * 4 * 3 * H * hd;
}
