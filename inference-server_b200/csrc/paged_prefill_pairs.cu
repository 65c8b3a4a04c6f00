// Tiled causal attention over KV pages for a chunk of prompt tokens on the tcgen05 tensor cores (sm_100a),
// head_dim 64 or 128, up to 128 query heads per kv head: the form with two tiles of rows in flight per CTA, for all but small calls,
// and the choice between it and paged_prefill_tc.cu.  Operation, arguments, row order and, row for row, the bits are the same there; what
// both replace in the reference is described in paged_prefill.cu (src/inference_server/kv_cache/hf_format.py:21-45 gather +
// src/inference_server/backends/torch_backend.py:107-147 chunk forward).
//
//   grid     A tile of rows is 128 rows of the score matrix: 128 / G consecutive prompt positions x the G query heads of a kv head.
//            The first `pairs` CTAs of a kv head own two neighbouring tiles, the others one; a CTA walks the key tiles (128 keys =
//            8 pages) of the context up to its last position.  Late positions (long walks) are issued first, of all kv heads side by
//            side (one kv head after the other leaves the last one's longest for the end: 2048 tokens from nothing 52 -> 42 us).
//   warp 0, warp 3   TMA producers: the Q tiles once, then per key tile the 8 K pages (warp 0) and V pages (warp 3) of the kv
//            head into two-stage rings.  A page (16 tokens) is one box of 8-row
//            swizzled atoms: a TMA copy costs about 100 cycles to issue whatever its size.
//   warp 1   score issuer (one thread): S = Q K^T of tile 0, then of tile 1, as 8 x tcgen05.mma M128 N128 K16 (kind::f16, bf16, both
//            operands K-major) into ONE accumulator: its 128 columns are read into registers at once (a thread owns a whole
//            row), so it is free again long before the row's exponentials are taken, and the next S is there when they are.
//   warp 2   P V issuer (one thread): O += P V as 2 x 4 tcgen05.mma M128 N128 K16, P (bf16, written by the
//            softmax warps) as the A operand from TMEM and V as an MN-major B operand straight from its page
//            layout [key][head_dim].  P is handed
//            over in two halves of 64 keys so that the first half's product runs while the second half's
//            exponentials are still being taken.
//   warps 4-7, 8-11   softmax of tile 0 and of tile 1, a thread per score row: tcgen05.ld of the row, causal mask by position, row
//            max, p = exp2((s - m) * scale) in fp32, P as bf16 into TMEM once the product of the key tile before has
//            finished.  The sums of a key tile's two halves are kept apart to the end.  The running max is lazy: O (in TMEM) and the running
//            sums are rescaled only when a row's max grew by more than 2^8 since the last rescale (any row
//            of the warp: the whole warp rescales, through tcgen05.ld / tcgen05.st, after the product of
//            the key tile before has finished); until then p is taken against the older max, which is exact
//            after the final division by the sum taken against the same max.
//   out      O / l as bf16, 256 contiguous bytes of a row per thread (128 in a CTA with one tile, whose idle softmax warps take half of
//            the columns).
//
// What bounds it: a key tile of one tile of rows is a chain (S -> maximum -> exponentials -> P -> product), and the special-function
// unit is busy 1180 of its cycles (1024 for the exponentials, the rest for the conversions of P, which share it); two tiles in
// flight fill each other's gaps and share K and V: 3000 cycles per key tile of both.  The other form, with one tile per CTA, two threads
// per row and P in shared memory, takes 2450 cycles per key tile of one.
// A wait on a barrier whose phase is long over still takes 200-300 cycles from a softmax warp, whose question queues behind
// exponentials.  So the two that rarely wait (P free, next S there) are asked without waiting in the middle of a half's
// exponentials (128 CTAs of 120 key tiles: 226 -> 206 us).
// us, the other form and this one, 32 / 4 heads of 128: 1024 tokens behind 14336 325, 217; 1500 behind 14001 476, 342; 2048 behind 8192 394, 255;
// 2048 from nothing 61.5, 41.6; 17 behind 14000 150, 133; one token 5.7, 6.0 (a row's
// exponentials are one thread's here).  16 / 2 heads of 64, 2048 behind 8192: 201, 147.
// What did not work: P over its own S, so that the next S waits for the product (4100 cycles per key tile of two); eight warps that
// share each tile and take them in turn (4400: nothing overlaps the maximum); a branch around the exponentials of a half that lies
// behind the warp's rows (one token 5.7, but 133 -> 147 us behind 14000).
//
// With 8 or 16 query heads per kv head the Q tiles come by TMA; with any other number G the softmax warps copy them
// (128 - 128 % G rows are used, the rest are zero rows that are never written out).
//
// Two run-time options, as in the decode kernel (paged_attn.cu): `chunk` > 0 cuts the sequence's positions into
// chunks counted from position 0, and a row sees only the keys of its own chunk - a tile's walk then begins at the
// key tile that holds the first key its first row sees, and a key tile's two mask edges (the row's chunk start, the row
// itself) are both per row; `gate` multiplies a row's output by the sigmoid of an fp32 number per (token, head).
// In this form a row may find its first key tiles fully masked: its running maximum stays -inf, its exponentials are taken
// against 0 (and are all 0), and the first key tile it does see rescales by 0 what is an exact 0.
//
// Registers: 168 per thread at launch, 224 in the softmax warps; the compiler keeps 36 to 44 bytes a thread in local memory (a row's 128
// scores and 32 words of P are live together).
// TMEM: O0, O1, S 128 columns each, P0, P1 64 (two bf16 per column).  Shared memory (head_dim 128): Q 2 x 32 KiB,
// K ring 2 x 32 KiB, V ring 2 x 32 KiB.  Every mbarrier wait is bounded; a wait that runs out records
// kErrDevWaitTimeout and the thread stops waiting but keeps the loop structure, so the kernel ends.

#include <algorithm>
#include <functional>
#include <utility>

#include "host.h"
#include "prefill_tc.cuh"

namespace b200 {

constexpr int kPairSoftmaxWarps = 8;
constexpr int kPairThreads = (4 + kPairSoftmaxWarps) * 32;
template <int D>
struct PairCfg {
  static constexpr int kTileBytes = D / 64 * kTcHalfBytes;  // Q, and one stage of K or V
  static constexpr int kRingBytes = 6 * kTileBytes;         // Q0, Q1, K0, K1, V0, V1
  static constexpr int kSmemBytes = kRingBytes + 1024 + 256 /* barriers, tmem base */ + kTcRows * 4 /* sums */;
};

// D[tmem] (+)= A[tmem] * B[smem], bf16: a lane of A is a row, a 32-bit column two neighbouring K elements.
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// G: query heads per kv head (8 or 16, Q tiles by TMA); 0 = `group` of them.
template <int D, int G>
__global__ void __launch_bounds__(kPairThreads, 1)
paged_attn_prefill_pairs_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                               const __grid_constant__ CUtensorMap v_map, const int* __restrict__ table_row,
                               __nv_bfloat16* __restrict__ out, int* __restrict__ err, int num_tokens, int first_pos,
                               int num_q_heads, int num_kv_heads, int num_blocks, float scale_log2, int group, int chunk, int pairs,
                               const float* __restrict__ gate, const __nv_bfloat16* __restrict__ q) {
#ifdef B200_DEVICE_OK
  constexpr int kTile = PairCfg<D>::kTileBytes;
  constexpr int kPageBytes = kTcPage * D * 2;
  constexpr uint32_t kAtomGroup = D / 64 * 1024;
  const int gr = G > 0 ? G : group;
  const int QT = kTcRows / gr;  // prompt positions per tile
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t q_sm = base, k_sm = base + 2 * kTile, v_sm = k_sm + 2 * kTile;
  const uint32_t bars = base + PairCfg<D>::kRingBytes;
  const uint32_t bar_kfull = bars, bar_kempty = bars + 16;       // [2 stages] each
  const uint32_t bar_vfull = bars + 32, bar_vempty = bars + 48;  // [2 stages] each
  const uint32_t bar_q = bars + 64;                              // [2 tiles] Q landed
  const uint32_t bar_sfull = bars + 80;                          // [2 tiles] S written, for this tile
  const uint32_t bar_odone = bars + 96;                          // [2 tiles] O += P V finished
  const uint32_t bar_pfull = bars + 112;                         // [2 tiles][2 halves of 64 keys] P written, O rescaled
  const uint32_t bar_sempty = bars + 144;                        // S read
  uint32_t* tmem_base_sm = reinterpret_cast<uint32_t*>(base_ptr + PairCfg<D>::kRingBytes + 192);

  float* l_sm = reinterpret_cast<float*>(base_ptr + PairCfg<D>::kRingBytes + 256);  // [128 rows]

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 32) {
    if (G > 0) tma_prefetch_desc(&q_map);
    tma_prefetch_desc(&k_map);
    tma_prefetch_desc(&v_map);
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(bar_kfull + 8 * s, 1);
      mbar_init(bar_kempty + 8 * s, 1);
      mbar_init(bar_vfull + 8 * s, 1);
      mbar_init(bar_vempty + 8 * s, 1);
      mbar_init(bar_q + 8 * s, G > 0 ? 1 : kPairSoftmaxWarps);
      mbar_init(bar_sfull + 8 * s, 1);
      mbar_init(bar_odone + 8 * s, 1);
      mbar_init(bar_pfull + 16 * s, 4);
      mbar_init(bar_pfull + 16 * s + 8, 4);
    }
    mbar_init(bar_sempty, 4);
    fence_mbar_init();
    fence_proxy_async();
  }
  if (warp == 1) tmem_alloc(smem_u32(tmem_base_sm), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_base_sm;
  const uint32_t tmem_o = tmem_base, tmem_s = tmem_base + 2 * kTcKeys, tmem_p = tmem_s + kTcKeys;  // O0, O1, S, P0, P1
  // late positions first, all kv heads of them side by side; the first `pairs` CTAs of a head take two tiles of rows each
  const int h = static_cast<int>(blockIdx.x) % num_kv_heads, cta = static_cast<int>(blockIdx.x) / num_kv_heads;
  const int own = cta < pairs ? 2 : 1;
  const int t0 = ((num_tokens + QT - 1) / QT - own - cta - min(cta, pairs)) * QT;
  const int t_end = min(t0 + own * QT, num_tokens);
  // key tiles that the CTA walks: from the first its first row sees to the one of its last row
  const int kt0 = first_visible(first_pos + t0 + 1, chunk) / kTcKeys;
  const int last_pos = first_pos + t_end - 1;
  const int n_tiles = last_pos / kTcKeys - kt0 + 1;
  // the part of the walk that a tile's rows see
  int tile_lo[2], tile_hi[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int first = t0 + t * QT;
    tile_lo[t] = tile_hi[t] = 0;
    if (first < t_end) {
      tile_lo[t] = first_visible(first_pos + first + 1, chunk) / kTcKeys - kt0;
      tile_hi[t] = (first_pos + min(first + QT, t_end) - 1) / kTcKeys - kt0 + 1;
    }
  }

  // Set-up done; Q and this chunk's K/V rows come from the kernel before this one.
  grid_dep_wait();
  grid_dep_launch();

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == 0 && G > 0) {
      if (lane < own) mbar_arrive_expect_tx(bar_q + 8 * lane, kTile);
      __syncwarp();
      // rows past the chunk are filled with zeros
      if (G == 8) {
        if (lane < own) tma_load_4d(q_sm + lane * kTile, &q_map, bar_q + 8 * lane, 0, h * 8, 0, t0 + lane * QT);
      } else if (lane < own * QT) {
        tma_load_4d(q_sm + lane * (G / 8) * kAtomGroup, &q_map, bar_q + 8 * (lane / QT), 0, 0, 0, ((t0 + lane) * num_q_heads + h * gr) / 8);
      }
    }
    if (warp == 0 || warp == 3) {
      // -------------------------------------------- K (warp 0), V (warp 3) ------
      // Lane i of the first 8 owns page i of a tile.
      const bool is_k = warp == 0;
      const uint32_t ring = is_k ? k_sm : v_sm, full = is_k ? bar_kfull : bar_vfull, empty = is_k ? bar_kempty : bar_vempty;
      const CUtensorMap* map = is_k ? &k_map : &v_map;
      const int pg = lane & 7, last_page = last_pos / kTcPage;
      bool alive = true;
#pragma unroll 1
      for (int j = 0; j < n_tiles; ++j) {
        const int st = j & 1;
        // pages past the last position hold nothing this CTA may read; the last valid page stands in so that
        // every stage is the same number of bytes and holds finite numbers (their scores are masked)
        int page = __ldg(table_row + min((kt0 + j) * kTcPages + pg, last_page));
        if (page < 0 || page >= num_blocks) {
          set_error(err, kErrDevBadBlockId);
          page = 0;
        }
        if (alive) alive = mbar_wait(empty + 8 * st, ((j >> 1) & 1) ^ 1, err);
        if (!__all_sync(0xffffffffu, alive)) break;
        if (lane == 0) mbar_arrive_expect_tx(full + 8 * st, kTile);
        __syncwarp();
        if (lane < kTcPages)
          tma_load_4d(ring + st * kTile + pg * kPageBytes, map, full + 8 * st, 0, 0, 0, (page * num_kv_heads + h) * (kTcPage / 8));
      }
    } else if (warp == 1) {
      // ------------------------------------------------- S = Q K^T ------
      if (elect_one()) {
        constexpr uint32_t idesc_s = tc_idesc_bf16(kTcRows, kTcKeys, 0);  // B = K, K-major
        bool alive = mbar_wait(bar_q, 0, err) && (own == 1 || mbar_wait(bar_q + 8, 0, err));
        uint32_t n = 0;
#pragma unroll 1
        for (int j = 0; j < n_tiles && alive; ++j) {
          const int st = j & 1;
          alive = mbar_wait(bar_kfull + 8 * st, (j >> 1) & 1, err);
          const uint64_t b0 = tc_desc_k_atoms(k_sm + st * kTile, kAtomGroup);
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (j < tile_lo[t] || j >= tile_hi[t]) continue;  // none of this tile's rows sees these keys
            if (alive) alive = mbar_wait(bar_sempty, (n & 1) ^ 1, err);
            if (!alive) break;
            ++n;
            tc_fence_after();
            const uint64_t a0 = tc_desc_k_atoms(q_sm + t * kTile, kAtomGroup);
#pragma unroll
            for (int k = 0; k < D / 16; ++k) {  // 16 of the head dimensions each
              const uint32_t off = ((k >> 2) * 1024 + (k & 3) * 32) >> 4;
              tc_mma_f16(tmem_s, a0 + off, b0 + off, idesc_s, k > 0 ? 1u : 0u);
            }
            tc_commit(bar_sfull + 8 * t);
          }
          tc_commit(bar_kempty + 8 * st);
        }
      }
    } else if (elect_one()) {
      // ------------------------------------------------- O += P V ------
      constexpr uint32_t idesc_o = tc_idesc_bf16(kTcRows, D, 1);  // B = V, MN-major
      bool alive = true;
#pragma unroll 1
      for (int j = 0; j < n_tiles && alive; ++j) {
        const int st = j & 1;
        alive = mbar_wait(bar_vfull + 8 * st, (j >> 1) & 1, err);
#pragma unroll
        for (int t = 0; t < 2; ++t) {
          if (j < tile_lo[t] || j >= tile_hi[t]) continue;
          const int i = j - tile_lo[t];
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            if (alive) alive = mbar_wait(bar_pfull + 16 * t + 8 * half, i & 1, err);
            if (!alive) break;
            tc_fence_after();
#pragma unroll
            for (int kk = half * 4; kk < half * 4 + 4; ++kk) {  // 16 keys each
              const uint64_t b = umma_desc_mn128(v_sm + st * kTile + kk * kPageBytes, 1024, kAtomGroup);
              tc_mma_f16_ts(tmem_o + t * kTcKeys, tmem_p + t * 64 + kk * 8, b, idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
            }
          }
          tc_commit(bar_odone + 8 * t);
        }
        tc_commit(bar_vempty + 8 * st);
      }
    }
  } else {
    // -------------------------------------------------------- softmax ------
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    const int t = (warp >> 2) - 1;           // tile of rows
    const int quarter = warp & 3;            // TMEM lanes this warp may touch
    const int r = quarter * 32 + lane;       // score row
    const uint32_t lane_off = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t s_acc = tmem_s + lane_off, o_acc = tmem_o + t * kTcKeys + lane_off, p_tm = tmem_p + t * 64 + lane_off;
    const uint32_t sfull = bar_sfull + 8 * t, odone = bar_odone + 8 * t, pfull = bar_pfull + 16 * t;
    const int tt0 = t0 + t * QT, rt = r / gr, n_own = t ? tile_hi[1] - tile_lo[1] : tile_hi[0] - tile_lo[0];
    const int pos = first_pos + min(tt0 + rt, min(tt0 + QT, num_tokens) - 1);  // the last key this row may see
    const int row_lo = first_visible(pos + 1, chunk);                          // and the first one
    if (G == 0) {  // copy the Q tiles: 16-byte pieces, neighbouring threads neighbouring pieces of a row
      for (int u = 0; u < own; ++u) {
        uint4 v[D / 16];
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const int i = threadIdx.x - 128 + k * 256, qr = i / (D / 8), qt_l = qr / gr, tok = t0 + u * QT + qt_l;
          v[k] = make_uint4(0u, 0u, 0u, 0u);
          if (qt_l < QT && tok < num_tokens)
            v[k] = *reinterpret_cast<const uint4*>(q + (static_cast<size_t>(tok) * num_q_heads + h * gr + (qr - qt_l * gr)) * D + i % (D / 8) * 8);
        }
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
          const int i = threadIdx.x - 128 + k * 256, qr = i / (D / 8), ch = i % (D / 8);
          *reinterpret_cast<uint4*>(base_ptr + u * kTile + (qr >> 3) * kAtomGroup + (ch >> 3) * 1024 + swz128(qr & 7, ch & 7)) = v[k];
        }
        fence_proxy_async();  // the tensor core reads Q through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_q + 8 * u);
      }
    }
    float m_run = -INFINITY, l_run[2] = {0.f, 0.f};  // the sums of the first and of the second halves of the key tiles
    bool alive = true, s_ready = false;
    int kbase = (kt0 + (t ? tile_lo[1] : tile_lo[0])) * kTcKeys;
#pragma unroll 1
    for (int i = 0; i < n_own; ++i, kbase += kTcKeys) {
      if (!__all_sync(0xffffffffu, s_ready) && alive) alive = mbar_wait(sfull, i & 1, err);
      tc_fence_after();
      float s[128];
      {
        uint32_t (&raw)[4][32] = *reinterpret_cast<uint32_t(*)[4][32]>(s);
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(s_acc + c * 32, raw[c]);
        tmem_ld_wait();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_sempty);  // S is the other tile's now
      if (kbase + kTcKeys - 1 > pos || kbase < row_lo) {  // the causal edge or the chunk's start runs through this row
#pragma unroll
        for (int c = 0; c < 128; ++c)
          if (kbase + c > pos || kbase + c < row_lo) s[c] = -INFINITY;
      }
      float mx4[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
      for (int c = 4; c < 124; c += 8)
#pragma unroll
        for (int k = 0; k < 4; ++k) mx4[k] = max3(mx4[k], s[c + k], s[c + 4 + k]);
#pragma unroll
      for (int k = 0; k < 4; ++k) mx4[k] = fmaxf(mx4[k], s[124 + k]);
      const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
      const bool need = (m_new - m_run) * scale_log2 > kTcRescaleLog2;  // true on the first tile (m_run = -inf)
      if (__any_sync(0xffffffffu, need)) {
        if (i > 0) {
          // O may be touched once the product of the tile before has finished
          if (alive) alive = mbar_wait(odone, (i - 1) & 1, err);
          tc_fence_after();
          // a row that has seen no key yet holds exact zeros
          const float alpha = m_new == -INFINITY ? 1.f : fast_exp2((m_run - m_new) * scale_log2);
          l_run[0] *= alpha;
          l_run[1] *= alpha;
#pragma unroll
          for (int c0 = 0; c0 < D; c0 += 32) {
            uint32_t o[32];
            tmem_ld32(o_acc + c0, o);
            tmem_ld_wait();
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * alpha);
            tmem_st32(o_acc + c0, o);
          }
        }
        m_run = m_new;
      }
      const float mb = m_run == -INFINITY ? 0.f : m_run * scale_log2;
      bool p_free = i == 0;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float sum4[4] = {0.f, 0.f, 0.f, 0.f};
        uint32_t pk[32];
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {
          // asked here, needed behind this half: P was last read by the product of the tile before; the next S
          if (ch == 5 && half == 0 && i > 0) p_free = mbar_test(odone, (i - 1) & 1);
          if (ch == 5 && half == 1) s_ready = mbar_test(sfull, (i + 1) & 1);
          float p[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) p[k] = fast_exp2(fmaf(s[half * 64 + ch * 8 + k], scale_log2, -mb));
          sum4[ch & 3] += ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
#pragma unroll
          for (int k = 0; k < 4; ++k) pk[ch * 4 + k] = pack_bf16x2(p[2 * k], p[2 * k + 1]);
        }
        l_run[half] += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
        if (half == 0 && !__all_sync(0xffffffffu, p_free) && alive) alive = mbar_wait(odone, (i - 1) & 1, err);
        tc_fence_after();
        tmem_st32(p_tm + half * 32, pk);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(pfull + 8 * half);
      }
    }
    // ---- epilogue: O / l, once the product of the last key tile has finished.  The warps of a CTA with one tile share its columns.
    const int e = own == 2 ? t : 0, cols = own == 2 ? D : D / 2, col0 = own == 2 ? 0 : t * (D / 2);
    float l = l_run[0] + l_run[1];
    if (own == 1) {
      if (t == 0) l_sm[r] = l;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      l = l_sm[r];
    }
    if (alive) alive = mbar_wait(bar_odone + 8 * e, (e ? tile_hi[1] - tile_lo[1] - 1 : tile_hi[0] - tile_lo[0] - 1) & 1, err);
    tc_fence_after();
    const int tok = t0 + e * QT + rt;
    const bool real = rt < QT && tok < t_end;
    const size_t oidx = static_cast<size_t>(tok) * num_q_heads + h * gr + (r - rt * gr);
    const float inv = (real ? head_gate(gate, oidx) : 1.f) / l;
    __nv_bfloat16* orow = out + oidx * D + col0;
#pragma unroll 1
    for (int c0 = 0; c0 < cols; c0 += 32) {
      uint32_t o[32];
      tmem_ld32(tmem_o + e * kTcKeys + lane_off + col0 + c0, o);
      tmem_ld_wait();
      if (real && alive) {
#pragma unroll
        for (int c = 0; c < 32; c += 8) {
          uint4 w;
          w.x = pack_bf16x2(__uint_as_float(o[c]) * inv, __uint_as_float(o[c + 1]) * inv);
          w.y = pack_bf16x2(__uint_as_float(o[c + 2]) * inv, __uint_as_float(o[c + 3]) * inv);
          w.z = pack_bf16x2(__uint_as_float(o[c + 4]) * inv, __uint_as_float(o[c + 5]) * inv);
          w.w = pack_bf16x2(__uint_as_float(o[c + 6]) * inv, __uint_as_float(o[c + 7]) * inv);
          *reinterpret_cast<uint4*>(orow + c0 + c) = w;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
#endif
}

// When the last CTA is done, in thirds of a single tile's key tile, if the first `pairs` CTAs of a kv head take two tiles of rows: every SM
// takes the next CTA in the order of the grid.  A key tile of two tiles of rows counts 4/3 of one of a single tile, and what a CTA
// does before and after its walk four key tiles.  Single tiles are priced as this file's; in the other form, which takes them in a call
// that sees few keys, a key tile costs a twentieth to an eighth more.
static int last_walk_end(int row_tiles, int pairs, int hkv, int qt, int first_pos, int num_tokens, int chunk, int sms) {
  using Free = std::pair<int, int>;  // a time, and how many SMs are free at it
  constexpr int kMost = 256;
  Free heap[kMost] = {{0, std::min(sms, kMost)}};
  int used = 1, end = 0;
  for (int c = 0, t = row_tiles; c < row_tiles - pairs; ++c) {
    const int tiles = c < pairs ? 2 : 1;
    t -= tiles;
    const int t0 = t * qt, last = first_pos + std::min(t0 + tiles * qt, num_tokens) - 1;
    const int first = chunk > 0 ? (first_pos + t0) / chunk * chunk : 0;
    const int length = (last / kTcKeys - first / kTcKeys + 1) * (tiles + 2) + 12;
    for (int left = hkv; left > 0;) {
      Free& next = heap[0];
      const int time = next.first, taken = std::min(next.second, left);
      next.second -= taken;
      if (next.second == 0) std::pop_heap(heap, heap + used--, std::greater<Free>());
      heap[used++] = {time + length, taken};
      std::push_heap(heap, heap + used, std::greater<Free>());
      end = std::max(end, time + length);
      left -= taken;
    }
  }
  return end;
}
// A call of single tiles that sees at most this many keys goes to the other form (paged_prefill_tc.cu).  Its loop is the slower one by
// 0.12 to 0.14 us per key tile of 128, but two threads share a row and its straight-line code is half as long, which a kernel that runs once per layer
// fetches anew each time: back to back both take 7.2 us for 91 tokens from nothing, and this form takes 33.7 -> 29.9 us for 91 tokens behind
// 2500 and 43.5 -> 39.3 behind 3500; in a whole pass (12 layers, us with the other form and with this one) 91 tokens from
// nothing take 2072, 2122, behind 2000 2393, 2414, behind 2900 2505, 2512, behind 3500 2578, 2576, behind 5000 2791, 2767; 300 tokens behind
// 2900 2740, 2745, behind 3500 2826, 2818; 17 tokens behind 3500 2138, 2146, behind 5000 2344, 2324.
constexpr int kSingleKeys = 3072;
// How many CTAs of a kv head take two tiles of rows.  None while every tile has an SM of its own (us, single tiles and pairs,
// 32 / 4 heads, 500 tokens behind 333, 128 tiles: 16.3, 18.6; 8 / 8 heads, 2048 behind 8192, 128 tiles: 121, 138).  With up to three
// tiles per SM the better of none and all by last_walk_end: over 678 calls of 600 to 4096 tokens, nine head counts, with and without
// chunks, the rule's choice is 0.3 percent behind the better form of each in the mean and 15 at worst, none 28 percent and all 0.8 (32 / 4
// heads from nothing: 600 tokens 13.9, 15.3; 1024 22.7, 21.3; 64 / 4 in chunks of 512, 1024 tokens 35.6, 24.9; 8 / 8, 3000 tokens 41.9, 46.7).
// Beyond that all (32 / 4, 2048 tokens 64, 42).
static int prefill_pairs(int row_tiles, int hkv, int qt, int first_pos, int num_tokens, int chunk, int sms) {
  if (row_tiles * hkv <= sms) return 0;
  const int all = row_tiles / 2;
  if (chunk == 0 && first_pos > num_tokens) {
    // Walks of about the same length come in waves, and a last wave of single tiles is a shorter one (1500 tokens behind 14001,
    // 376 tiles: two waves of pairs 413 us, 148 pairs and 80 single tiles 342).
    const int pairs = std::min(all, row_tiles * hkv / (2 * sms) * sms / hkv);
    return (row_tiles - 2 * pairs) * hkv <= sms ? pairs : all;
  }
  if (row_tiles * hkv > 3 * sms) return all;
  const int two = last_walk_end(row_tiles, all, hkv, qt, first_pos, num_tokens, chunk, sms);
  return two < last_walk_end(row_tiles, 0, hkv, qt, first_pos, num_tokens, chunk, sms) ? all : 0;
}

// How a call is laid out: tiles of 128 score rows per kv head, how many CTAs of a head take two of them, and whether its single tiles go to
// the other form.
struct PrefillPlan {
  int row_tiles, pairs;
  bool other_form;
};
static PrefillPlan prefill_plan(int num_tokens, int first_pos, int hq, int hkv, int chunk, int sms) {
  PrefillPlan p;
  const int qt = kTcRows / (hq / hkv), keys = first_pos + num_tokens;
  p.row_tiles = (num_tokens + qt - 1) / qt;
  p.pairs = prefill_pairs(p.row_tiles, hkv, qt, first_pos, num_tokens, chunk, sms);
  p.other_form = p.pairs == 0 && (chunk > 0 ? std::min(chunk, keys) : keys) <= kSingleKeys;
  return p;
}

template <int D, int G>
static int launch_prefill_pairs_g(const CUtensorMap& qmap, const CUtensorMap& kmap, const CUtensorMap& vmap, const void* q,
                                  const int* table_row, void* out, int* err, int num_tokens, int first_pos, int hq, int hkv,
                                  int num_blocks, float scale, int chunk, const float* gate, cudaStream_t st, int row_tiles, int pairs) {
  int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(&paged_attn_prefill_pairs_kernel<D, G>), PairCfg<D>::kSmemBytes);
  if (rc) return rc;
  B200_CUDA(launch_overlapped(paged_attn_prefill_pairs_kernel<D, G>, dim3((row_tiles - pairs) * hkv), dim3(kPairThreads),
                              PairCfg<D>::kSmemBytes, st, qmap, kmap, vmap, table_row, static_cast<__nv_bfloat16*>(out), err,
                              num_tokens, first_pos, hq, hkv, num_blocks, scale * 1.4426950408889634f, hq / hkv, chunk, pairs, gate,
                              static_cast<const __nv_bfloat16*>(q)));
  return 0;
}

// paged_prefill_tc.cu
int launch_prefill_single(const CUtensorMap& qmap, const CUtensorMap& kmap, const CUtensorMap& vmap, bool q_tma, int head_dim, const void* q,
                          const int* table_row, void* out, int* err, int num_tokens, int first_pos, int hq, int hkv, int num_blocks,
                          float scale, int chunk, const float* gate, cudaStream_t st);

// The tcgen05 form of the prompt attention: head_dim 64 or 128, 1 to 128 query heads per kv head, at most 65535 kv
// heads, q and out 16-byte aligned.  Arguments as launch_prefill in paged_prefill.cu, which has checked them.
int launch_prefill_tc(const void* q, const void* k_pool, const void* v_pool, const int* table_row, void* out, int* err,
                      int num_tokens, int first_pos, int hq, int hkv, int head_dim, int num_blocks, float scale,
                      int chunk, const float* gate, cudaStream_t st) {
  const int group = hq / hkv;
  CUtensorMap qmap, kmap, vmap;
  const uint64_t rows = static_cast<uint64_t>(num_blocks) * hkv * kTcPage;
  int rc = get_tensor_map_atoms(k_pool, rows, head_dim, kTcPage, &kmap);
  if (rc) return rc;
  rc = get_tensor_map_atoms(v_pool, rows, head_dim, kTcPage, &vmap);
  if (rc) return rc;
  const bool q_tma = head_dim == 128 && (group == 8 || group == 16);
  if (q_tma) {
    // 8 query heads per kv head: the CTA's positions in one box; 16: a box per position
    rc = group == 8 ? get_tensor_map_atoms_of(q, num_tokens, hq, head_dim, kTcRows / 8, &qmap)
                    : get_tensor_map_atoms(q, static_cast<uint64_t>(num_tokens) * hq, head_dim, 16, &qmap);
    if (rc) return rc;
  } else {
    qmap = kmap;  // not read
  }
  int sms = 0;
  rc = device_sm_count(&sms);
  if (rc) return rc;
  const PrefillPlan plan = prefill_plan(num_tokens, first_pos, hq, hkv, chunk, sms);
  const int row_tiles = plan.row_tiles, pairs = plan.pairs;
  if (plan.other_form)
    return launch_prefill_single(qmap, kmap, vmap, q_tma, head_dim, q, table_row, out, err, num_tokens, first_pos, hq, hkv, num_blocks,
                                 scale, chunk, gate, st);
#define B200_TC_ARGS qmap, kmap, vmap, q, table_row, out, err, num_tokens, first_pos, hq, hkv, num_blocks, scale, chunk, \
                     gate, st, row_tiles, pairs
  if (q_tma && group == 8) return launch_prefill_pairs_g<128, 8>(B200_TC_ARGS);
  if (q_tma) return launch_prefill_pairs_g<128, 16>(B200_TC_ARGS);
  if (head_dim == 128) return launch_prefill_pairs_g<128, 0>(B200_TC_ARGS);
  return launch_prefill_pairs_g<64, 0>(B200_TC_ARGS);
#undef B200_TC_ARGS
}

}  // namespace b200

using namespace b200;

extern "C" int b200_paged_attn_prefill_pairs(int num_tokens, int first_position, int num_q_heads, int num_kv_heads, int chunk, int num_sms,
                                             int* short_form) {
  B200_REQUIRE(num_tokens > 0 && first_position >= 0 && num_kv_heads > 0 && num_q_heads % num_kv_heads == 0 && num_q_heads > 0 &&
                   num_q_heads / num_kv_heads <= kTcRows && chunk >= 0 && num_sms > 0,
               "paged_attn_prefill_pairs: %d tokens from %d, %d query heads over %d, chunk %d, %d SMs", num_tokens, first_position, num_q_heads,
               num_kv_heads, chunk, num_sms);
  const PrefillPlan plan = prefill_plan(num_tokens, first_position, num_q_heads, num_kv_heads, chunk, num_sms);
  if (short_form != nullptr) *short_form = plan.other_form;
  return plan.pairs;
}
