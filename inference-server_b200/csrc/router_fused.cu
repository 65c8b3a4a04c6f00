// Residual add + RMSNorm + router projection + top-k routing in one kernel (sm_100a).
//
// In the reference's model forward (src/inference_server/backends/torch_backend.py:314-320 ->
// transformers Qwen3MoeDecoderLayer / Qwen3MoeSparseMoeBlock) these are a residual add, the
// post-attention RMSNorm, the router's linear layer `gate` and Qwen3MoeTopKRouter (fp32 softmax,
// top-k, renormalisation): four dependent launches that move a few megabytes.  At decode sizes
// their cost is launch and memory latency, not bandwidth, so they are fused here:
//
//   x += delta (bf16);  h = weight * rmsnorm(x);  logits = h W_r^T (fp32);  ids, weights = top-k
//
//   grid   = (rows / ROWS) clusters of 8 CTAs.  A cluster owns ROWS = 16 rows, or 32 where that saves
//            enough waves of clusters (route_rows); CTA r of it owns the r-th
//            eighth of the hidden dimension, so the router matrix [E, H] (0.5 MiB at E = 128,
//            H = 2048, too much for one CTA to pull in time) is read as eight 64 KiB slices.
//   norm   = each CTA adds and squares its slice of the rows; the eight partial sums of squares
//            meet through distributed shared memory (ROWS floats per CTA) and are added in rank order.
//   gemm   = [ROWS x H/8] x [H/8 x E] per CTA by mma.sync m16n8k16 (bf16 in, fp32 out): 134 MFLOP for
//            256 rows, far too little for the tcgen05 path to pay its set-up; warp w takes experts
//            16w..16w+15.  The eight partial logit tiles (ROWS x E fp32) meet through distributed
//            shared memory: CTA r sums rows ROWS/8 * r ... in rank order.
//   route  = those rows are routed by a warp each exactly as moe_route_kernel does (selection on
//            the logits, ties to the lower expert id), on fp32 logits that never leave the chip.
// What bounds it is a chain of dependent waits, so each step asks for all it needs at once: the rows a warp adds, the fragments of
// several MMA steps, and the top-k is two warp reductions per round (warp_topk, common.cuh).  128 experts of width 2048, us before and
// now: 1 row 8.0, 5.0   256: 10.1, 6.9   1024: 14.6, 11.1   2048: 28.6, 21.6.  (A form without clusters, the router matrix streamed
// through each CTA for 16 rows, took 22.4 at 2048 rows and 18.8 at one.)
// Everything is deterministic (fixed summation orders, no atomics).

#include <mutex>

#include "common.cuh"
#include "host.h"

namespace b200 {

constexpr int kRfCluster = 8;    // CTAs per cluster = slices of the hidden dimension
constexpr int kRfThreads = 256;
constexpr int kRfMaxExperts = 128;

__device__ __forceinline__ uint32_t rf_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void rf_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float rf_ld_peer(const float* local, uint32_t rank) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local)), "r"(rank));
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote));
  return v;
}
__device__ __forceinline__ void rf_cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

struct RouterFusedParams {
  __nv_bfloat16* x;             // [T, H] residual stream, updated in place when delta is given
  const __nv_bfloat16* delta;   // [T, H] or null
  const __nv_bfloat16* norm_w;  // [H]
  const __nv_bfloat16* router;  // [E, H]
  __nv_bfloat16* normed;        // [T, H]
  int* topk_ids;                // [T, K]
  float* topk_w;                // [T, K]
  float* logits_out;            // [T, E] or null
  const int* num_valid;         // device scalar or null
  float eps;
  int T, H, E, K, renorm;
};

// Top-k of a row by a warp (the arithmetic of moe_route_kernel) from its fp32 logits in shared memory.
__device__ __forceinline__ void rf_route_row(const RouterFusedParams& p, int row, const float* lg, int lane) {
  const int E = p.E, K = p.K;
  if (p.num_valid != nullptr && row >= *p.num_valid) {
    if (lane < K) {
      p.topk_ids[static_cast<size_t>(row) * K + lane] = -1;
      p.topk_w[static_cast<size_t>(row) * K + lane] = 0.f;
    }
    return;
  }
  constexpr int kPer = kRfMaxExperts / 32;
  float v[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const int e = lane + 32 * j;
    v[j] = e < E ? lg[e] : -INFINITY;
  }
  float mine;
  int my_id;
  warp_topk<kPer>(v, E, K, lane, &mine, &my_id);
  const float mx = __shfl_sync(0xffffffffu, mine, 0);
  const float my_p = expf(mine - mx);
  float den = 0.f;
  if (p.renorm) {
    den = lane_sum_in_order(my_p, K);
  } else {
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (lane + 32 * j < E) den += expf(v[j] - mx);
    den = warp_sum(den);
  }
  if (lane < K) {
    p.topk_ids[static_cast<size_t>(row) * K + lane] = my_id;
    p.topk_w[static_cast<size_t>(row) * K + lane] = my_p / den;
  }
}

// (four CTAs of the 16-row form per SM, three of the 32-row form: where shared memory allows so many, registers must not forbid them)
template <int ROWS>
__global__ void __launch_bounds__(kRfThreads, ROWS == 16 ? 4 : 3)
add_rmsnorm_route_kernel(const RouterFusedParams p) {
#ifdef B200_DEVICE_OK
  extern __shared__ __align__(16) uint8_t rf_smem[];
  constexpr int kOwn = ROWS / kRfCluster;  // rows a CTA finishes; also rows per warp of the norm
  const int cols = p.H / kRfCluster;       // this CTA's slice of the hidden dimension
  const int pitch = cols + 8;              // bf16 elements per smem row: 16 bytes of padding keep ldmatrix conflict-free
  __nv_bfloat16* a_tile = reinterpret_cast<__nv_bfloat16*>(rf_smem);   // [ROWS][pitch]
  __nv_bfloat16* w_tile = a_tile + ROWS * pitch;                     // [E][pitch]
  float* ss_part = reinterpret_cast<float*>(w_tile + static_cast<size_t>(p.E) * pitch);  // [ROWS]
  float* inv_sm = ss_part + ROWS;                                       // [ROWS]
  float* lg_part = inv_sm + ROWS;                                       // [ROWS][E]
  float* lg_fin = lg_part + ROWS * p.E;                                 // [kOwn][E]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = rf_cluster_rank();
  const int row0 = (static_cast<int>(blockIdx.x) / kRfCluster) * ROWS;
  const int col0 = static_cast<int>(rank) * cols;

  // ---- the router slice [E][cols] starts flowing into shared memory right away
  {
    const int chunks_per_row = cols / 8;  // 16-byte pieces
    const int total = p.E * chunks_per_row;
    for (int i = tid; i < total; i += kRfThreads) {
      const int e = i / chunks_per_row, c = i - e * chunks_per_row;
      rf_cp_async16(smem_u32(w_tile + static_cast<size_t>(e) * pitch + c * 8),
                    p.router + static_cast<size_t>(e) * p.H + col0 + c * 8);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // (a lane's first piece of the norm weights too)
  uint4 wfirst = make_uint4(0u, 0u, 0u, 0u);
  if (lane < cols / 8) wfirst = *reinterpret_cast<const uint4*>(p.norm_w + col0 + lane * 8);
  // The router matrix and the norm's weights are weights; the rows come from the kernels before this one.
  grid_dep_wait();
  grid_dep_launch();

  // ---- residual add, partial sums of squares: warp w owns rows kOwn * w ..., whose loads are in flight together
  float ss[kOwn];
#pragma unroll
  for (int rr = 0; rr < kOwn; ++rr) ss[rr] = 0.f;
  for (int c = lane; c < cols / 8; c += 32) {
    uint4 xv[kOwn], dv[kOwn];
#pragma unroll
    for (int rr = 0; rr < kOwn; ++rr) {
      const int row = row0 + kOwn * warp + rr;
      const size_t off = static_cast<size_t>(row) * p.H + col0 + c * 8;
      xv[rr] = dv[rr] = make_uint4(0u, 0u, 0u, 0u);
      if (row < p.T) {
        xv[rr] = *reinterpret_cast<const uint4*>(p.x + off);
        if (p.delta != nullptr) dv[rr] = *reinterpret_cast<const uint4*>(p.delta + off);
      }
    }
#pragma unroll
    for (int rr = 0; rr < kOwn; ++rr) {
      const int r = kOwn * warp + rr, row = row0 + r;
      uint4 raw = xv[rr];
      if (row < p.T) {
        __nv_bfloat162* h2 = reinterpret_cast<__nv_bfloat162*>(&raw);
        if (p.delta != nullptr) {
          const __nv_bfloat162* d2 = reinterpret_cast<const __nv_bfloat162*>(&dv[rr]);
#pragma unroll
          for (int j = 0; j < 4; ++j) h2[j] = __hadd2(h2[j], d2[j]);  // the residual add happens in bf16, as in the model
          *reinterpret_cast<uint4*>(p.x + static_cast<size_t>(row) * p.H + col0 + c * 8) = raw;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(h2[j]);
          ss[rr] += f.x * f.x + f.y * f.y;
        }
      }
      *reinterpret_cast<uint4*>(a_tile + r * pitch + c * 8) = raw;
    }
  }
#pragma unroll
  for (int rr = 0; rr < kOwn; ++rr) {
    const float sum = warp_sum(ss[rr]);
    if (lane == 0) ss_part[kOwn * warp + rr] = sum;
  }
  __syncwarp();
  rf_cluster_sync();  // #1: every slice's partial sums are written
  if (tid < ROWS) {
    float part[kRfCluster];
#pragma unroll
    for (int pr = 0; pr < kRfCluster; ++pr) part[pr] = rf_ld_peer(ss_part + tid, pr);
    float tot = 0.f;
#pragma unroll
    for (int pr = 0; pr < kRfCluster; ++pr) tot += part[pr];
    inv_sm[tid] = rsqrtf(tot / static_cast<float>(p.H) + p.eps);
  }
  __syncthreads();

  // ---- normalise: out = weight * bf16(x * inv); kept in shared memory as the A operand, written out as h
  for (int c = lane; c < cols / 8; c += 32) {
    const uint4 wraw = c == lane ? wfirst : *reinterpret_cast<const uint4*>(p.norm_w + col0 + c * 8);
    const __nv_bfloat162* w2 = reinterpret_cast<const __nv_bfloat162*>(&wraw);
#pragma unroll
    for (int rr = 0; rr < kOwn; ++rr) {
      const int r = kOwn * warp + rr, row = row0 + r;
      const float inv = inv_sm[r];
      uint4 raw = *reinterpret_cast<const uint4*>(a_tile + r * pitch + c * 8);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
      uint4 o;
      __nv_bfloat162* o2 = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h2[j]);
        o2[j] = __hmul2(w2[j], __floats2bfloat162_rn(f.x * inv, f.y * inv));
      }
      *reinterpret_cast<uint4*>(a_tile + r * pitch + c * 8) = o;
      if (row < p.T) *reinterpret_cast<uint4*>(p.normed + static_cast<size_t>(row) * p.H + col0 + c * 8) = o;
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- partial logits of this slice: warp w takes experts 16w .. 16w + 15
  if (warp * 16 < p.E) {
    constexpr int kMt = ROWS / 16;
    float acc[kMt][2][4];
#pragma unroll
    for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = acc[mt][nt][2] = acc[mt][nt][3] = 0.f;
    const int mat = lane >> 3, lr = lane & 7;
    const uint32_t a_addr = smem_u32(a_tile) + static_cast<uint32_t>(((mat & 1) * 8 + lr) * pitch * 2 + (mat >> 1) * 16);
    const uint32_t b_addr =
        smem_u32(w_tile) + static_cast<uint32_t>((warp * 16 + (mat >> 1) * 8 + lr) * pitch * 2 + (mat & 1) * 16);
    // the fragments of kStep steps are in flight together (a slice is a multiple of 64 columns)
    constexpr int kStep = ROWS == 16 ? 4 : 2;
    for (int k0 = 0; k0 < cols / 16; k0 += kStep) {
      uint32_t b[kStep][4], a[kStep][kMt][4];
#pragma unroll
      for (int k = 0; k < kStep; ++k) {
        ldmatrix_x4(b_addr + (k0 + k) * 32, b[k][0], b[k][1], b[k][2], b[k][3]);
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt)
          ldmatrix_x4(a_addr + mt * 16 * pitch * 2 + (k0 + k) * 32, a[k][mt][0], a[k][mt][1], a[k][mt][2], a[k][mt][3]);
      }
#pragma unroll
      for (int k = 0; k < kStep; ++k)
#pragma unroll
        for (int mt = 0; mt < kMt; ++mt) {
          mma_bf16_16816(acc[mt][0], a[k][mt], b[k][0], b[k][1]);
          mma_bf16_16816(acc[mt][1], a[k][mt], b[k][2], b[k][3]);
        }
    }
    const int gq = lane >> 2, tq = lane & 3;
#pragma unroll
    for (int mt = 0; mt < kMt; ++mt)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        float* lo = lg_part + (mt * 16 + gq) * p.E + warp * 16 + nt * 8 + 2 * tq;
        lo[0] = acc[mt][nt][0];
        lo[1] = acc[mt][nt][1];
        lo[8 * p.E] = acc[mt][nt][2];
        lo[8 * p.E + 1] = acc[mt][nt][3];
      }
  }
  __syncwarp();
  rf_cluster_sync();  // #2: every slice's partial logits are written

  // ---- CTA r finishes rows kOwn * r ...: slices summed in rank order
#pragma unroll
  for (int r0 = 0; r0 < kOwn; r0 += 2) {
    const int rl = r0 + (tid >> 7), e = tid & 127;  // 256 threads = 2 rows x up to 128 experts
    if (e < p.E) {
      const int r = kOwn * static_cast<int>(rank) + rl;
      float part[kRfCluster];
#pragma unroll
      for (int pr = 0; pr < kRfCluster; ++pr) part[pr] = rf_ld_peer(lg_part + r * p.E + e, pr);
      float tot = 0.f;
#pragma unroll
      for (int pr = 0; pr < kRfCluster; ++pr) tot += part[pr];
      lg_fin[rl * p.E + e] = tot;
      const int row = row0 + r;
      if (p.logits_out != nullptr && row < p.T) p.logits_out[static_cast<size_t>(row) * p.E + e] = tot;
    }
  }
  __syncthreads();

  // ---- top-k of these rows (the arithmetic of moe_route_kernel)
  if (warp < kOwn) {
    const int row = row0 + kOwn * static_cast<int>(rank) + warp;
    if (row < p.T) rf_route_row(p, row, lg_fin + warp * p.E, lane);
  }
  __syncwarp();
  rf_cluster_sync();  // #3: nobody leaves while a peer may still read its shared memory
#endif
}

static size_t router_fused_smem(int H, int E, int rows) {
  const size_t pitch = static_cast<size_t>(H) / kRfCluster + 8;
  return (rows + static_cast<size_t>(E)) * pitch * 2 + (2 * rows + rows * static_cast<size_t>(E) + rows / kRfCluster * E) * 4;
}

static void route_launch_config(cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, int clusters, size_t smem, cudaStream_t st) {
  *cfg = cudaLaunchConfig_t{};
  cfg->gridDim = dim3(static_cast<unsigned>(clusters) * kRfCluster);
  cfg->blockDim = dim3(kRfThreads);
  cfg->dynamicSmemBytes = smem;
  cfg->stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kRfCluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr;
  cfg->numAttrs = 1;
}

template <int ROWS>
static int launch_route(const RouterFusedParams& p, cudaStream_t st) {
  const size_t smem = router_fused_smem(p.H, p.E, ROWS);
  int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(&add_rmsnorm_route_kernel<ROWS>), static_cast<int>(smem));
  if (rc) return rc;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[2];
  route_launch_config(&cfg, attr, (p.T + ROWS - 1) / ROWS, smem, st);
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  if (overlapped_launch_enabled()) cfg.numAttrs = 2;
  B200_CUDA(cudaLaunchKernelEx(&cfg, add_rmsnorm_route_kernel<ROWS>, p));
  return 0;
}

// How many clusters of ROWS rows the current device holds at once; asked once per device and size of shared memory.
template <int ROWS>
static int resident_route_clusters(int H, int E, int* out) {
  struct Entry {
    int dev;
    size_t smem;
    int n;
  };
  static std::mutex mu;
  static Entry cache[32];
  static int used = 0;
  const size_t smem = router_fused_smem(H, E, ROWS);
  int dev = 0;
  B200_CUDA(cudaGetDevice(&dev));
  {
    std::lock_guard<std::mutex> lock(mu);
    for (int i = 0; i < used; ++i)
      if (cache[i].dev == dev && cache[i].smem == smem) {
        *out = cache[i].n;
        return 0;
      }
  }
  int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(&add_rmsnorm_route_kernel<ROWS>), static_cast<int>(smem));
  if (rc) return rc;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  route_launch_config(&cfg, attr, 1, smem, nullptr);
  int n = 0;
  B200_CUDA(cudaOccupancyMaxActiveClusters(&n, add_rmsnorm_route_kernel<ROWS>, &cfg));
  if (n < 1) n = 1;
  std::lock_guard<std::mutex> lock(mu);
  if (used < static_cast<int>(sizeof(cache) / sizeof(cache[0]))) cache[used++] = Entry{dev, smem, n};
  *out = n;
  return 0;
}

// Rows per cluster: 16, or 32 where their waves take less.  A wave of 32-row clusters takes at most 1.15 times one of 16-row clusters, and how many
// of either the GPU holds depends on their shared memory, so on width and experts.  us with 16 and with 32, and the waves of each:
//   128 experts, width  512  1024 rows 9.2, 10.2   2048: 16.9, 17.4 (2, 2)   4096: 31.3, 28.2 (4, 3)   5000: 38.0, 34.4 (5, 4)
//   128 experts, width 2048   513 rows 8.8, 9.8    1024: 16.8, 11.3 (2, 1)   2048: 32.1, 21.6 (4, 2)
//   128 experts, width 4096   256 rows 14.7, 9.5    512: 22.8, 18.6         1024: 39.6, 29.1 (5, 3)
//    64 experts, width 2048  5000 rows 42.0, 37.3 (5, 4)   6000: 49.8, 41.8 (6, 4)
static int route_rows(int T, int H, int E, int* out) {
  *out = 16;
  const int c16 = (T + 15) / 16, c32 = (T + 31) / 32;
  if (c16 < 2 || router_fused_smem(H, E, 32) > 200 * 1024) return 0;
  int n16 = 0, n32 = 0;
  int rc = resident_route_clusters<16>(H, E, &n16);
  if (rc) return rc;
  if (c16 <= n16) return 0;
  rc = resident_route_clusters<32>(H, E, &n32);
  if (rc) return rc;
  if (23 * ((c32 + n32 - 1) / n32) <= 20 * ((c16 + n16 - 1) / n16)) *out = 32;
  return 0;
}

}  // namespace b200

using namespace b200;

extern "C" int b200_add_rmsnorm_route_supported(int hidden, int num_experts, int top_k) {
  return hidden > 0 && hidden % (kRfCluster * 64) == 0 && num_experts > 0 && num_experts % 16 == 0 &&
         num_experts <= kRfMaxExperts && top_k > 0 && top_k <= 32 && top_k <= num_experts &&
         router_fused_smem(hidden, num_experts, 16) <= 200 * 1024;
}

extern "C" int b200_add_rmsnorm_route(void* x, const void* delta, const void* norm_weight, float eps,
                                      const void* router_weight, int num_rows, int hidden, int num_experts,
                                      int top_k, int renormalize, const int32_t* num_valid_rows, void* normed_out,
                                      int32_t* topk_ids, float* topk_weights, float* logits_out, void* stream) {
  B200_REQUIRE(x && norm_weight && router_weight && normed_out && topk_ids && topk_weights,
               "add_rmsnorm_route: null pointer");
  B200_REQUIRE(num_rows >= 0, "add_rmsnorm_route: negative row count");
  B200_REQUIRE(b200_add_rmsnorm_route_supported(hidden, num_experts, top_k),
               "add_rmsnorm_route: hidden %d must be a multiple of 512, num_experts %d a multiple of 16 and at most "
               "%d, top_k %d at most min(32, num_experts)", hidden, num_experts, kRfMaxExperts, top_k);
  B200_REQUIRE(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(delta) |
                 reinterpret_cast<uintptr_t>(norm_weight) | reinterpret_cast<uintptr_t>(router_weight) |
                 reinterpret_cast<uintptr_t>(normed_out)) & 15) == 0,
               "add_rmsnorm_route: buffers must be 16-byte aligned");
  int rc = check_device(nullptr);
  if (rc) return rc;
  if (num_rows == 0) return 0;
  RouterFusedParams p{};
  p.x = static_cast<__nv_bfloat16*>(x);
  p.delta = static_cast<const __nv_bfloat16*>(delta);
  p.norm_w = static_cast<const __nv_bfloat16*>(norm_weight);
  p.router = static_cast<const __nv_bfloat16*>(router_weight);
  p.normed = static_cast<__nv_bfloat16*>(normed_out);
  p.topk_ids = topk_ids;
  p.topk_w = topk_weights;
  p.logits_out = logits_out;
  p.num_valid = num_valid_rows;
  p.eps = eps;
  p.T = num_rows;
  p.H = hidden;
  p.E = num_experts;
  p.K = top_k;
  p.renorm = renormalize;
  int rows = 16;
  rc = route_rows(num_rows, hidden, num_experts, &rows);
  if (rc) return rc;
  return rows == 32 ? launch_route<32>(p, as_stream(stream)) : launch_route<16>(p, as_stream(stream));
}

extern "C" int b200_add_rmsnorm_route_rows(int num_rows, int hidden, int num_experts) {
  B200_REQUIRE(num_rows > 0 && b200_add_rmsnorm_route_supported(hidden, num_experts, 1), "add_rmsnorm_route_rows: %d rows of %d, %d experts",
               num_rows, hidden, num_experts);
  int rc = check_device(nullptr);
  if (rc) return rc;
  int rows = 0;
  rc = route_rows(num_rows, hidden, num_experts, &rows);
  return rc ? rc : rows;
}
