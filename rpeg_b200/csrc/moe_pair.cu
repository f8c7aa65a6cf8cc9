// Grouped GEMM of a mixture of experts for prompts: two CTAs on a tile (tcgen05 cta_group::2) with the weights on the M axis.
//
//   C[r, 0..N) = act( A[r, 0..K) * B_s[0..N, 0..K)^T )   for every row r of segment s (operands and segments as in moe.cu)
//
// An expert's rows are any number, and a tile of 128 or 256 rows is computed whole: at 500 rows an expert a seventh to a third of
// the work was padding. Here a tile is 256 features x bn tokens, and bn is the segment's own: its rows in as few tiles as hold 256
// each, equal ones, a multiple of 32. The pair halves what an SM reads of either operand (gemm_pair.cu). What is left of padding is the
// last tile of features (1408: 8 %).
// Bound by the tensor cores; 8000 tokens, 6 of 64 experts: gated 1024 x 4096 683 us with 128-row tiles, now 607 (1.33
// PFLOP/s); 4096 x 1024 378 and 300 us; 5800 tokens and two always-on experts, 4096 x 1408 501 and 421 us.
//
// The accumulator is transposed (lane = feature, column = token): every epilogue warp turns 32 x 32 outputs through its own staging
// buffer and stores whole 64-byte (gated: 32-byte) pieces of rows, those of the segment only.
// Gated: the rows of the weight tile alternate, 16 gate rows, 16 up rows of the same features, so that a lane finds its other half 16 lanes
// away in its own warp. A tensor map of [experts][groups of 16][gate, up][16 rows][K] brings them in that order in one box (eight
// boxes of 16 rows: half the speed).
#include "act_io.cuh"
#include "moe_segments.cuh"
#include "pair.cuh"
#include "rpeg_kernels.h"

namespace rpeg {

constexpr int MP_MAX_SEGMENTS = 1024;
constexpr int MP_BK = 64, MP_STAGES = 6, MP_THREADS = 192;
constexpr int MP_HALF_BYTES = 128 * MP_BK * 2;             // 128 weight rows; 128 token rows
constexpr int MP_STAGE_BYTES = 2 * MP_HALF_BYTES;
constexpr int MP_STAGING = 4 * 2048;
constexpr int MP_SMEM = 1024 + MP_STAGES * MP_STAGE_BYTES + MP_STAGING + 512 + (MP_MAX_SEGMENTS + 1) * 4;
static_assert(MP_SMEM <= 227 * 1024, "shared memory");

template <int ACT>
__global__ void __launch_bounds__(MP_THREADS, 1) __cluster_dims__(2, 1, 1)
moe_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_b,
                __nv_bfloat16* __restrict__ C, const int* __restrict__ seg_off, int n_routed, int n_shared, int seg_rows, int shared_from_x, int N,
                int K, int ldc, int* status) {
  constexpr bool GATED = ACT == FF_SWIGLU;
  constexpr int TF = GATED ? 128 : 256;                    // features per tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + MP_STAGES * MP_STAGE_BYTES;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(staging + MP_STAGING);     // even CTA: both CTAs' bytes of a stage
  uint64_t* empty_bar = full_bar + MP_STAGES;                                 // each CTA: the pair's MMAs have read the stage
  uint64_t* tfull_bar = empty_bar + MP_STAGES;                                // each CTA: accumulator complete
  uint64_t* tempty_bar = tfull_bar + 2;                                       // even CTA: all eight epilogue warps have read it
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* first_tile = reinterpret_cast<int*>(staging + MP_STAGING + 512);       // [segments + 1] token tiles before a segment

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_rank());
  const int S = n_routed + n_shared;
  if (threadIdx.x == 0) {
    for (int s = 0; s < MP_STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], 8);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_x);
    tma_prefetch_desc(&tmap_b);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  griddep_launch();
  griddep_wait();
  if (warp == 2) {
    int carry = 0;
    for (int s0 = 0; s0 < S; s0 += 32) {
      const int s = s0 + lane;
      int v = s < S ? (moe_segment(seg_off, n_routed, seg_rows, s).rows + 255) / 256 : 0;
      const int own = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
      }
      if (s < S) first_tile[s] = carry + v - own;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
    if (lane == 0) first_tile[S] = carry;
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();                   // the other CTA's barriers exist before anything is counted on them
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int f_tiles = (N + TF - 1) / TF;
  const int num_items = first_tile[S] * f_tiles;
  const int num_kb = (K + MP_BK - 1) / MP_BK;
  const int first = blockIdx.x >> 1, step = gridDim.x >> 1;

  // Items of a segment: its token tiles vary fastest, so the pairs that run side by side share a weight tile.
  struct Item { int seg, f0, t0, bn, rows; long long row0; };        // tokens [t0, t0 + rows) of the segment, which starts at row0
  auto item = [&](int w) -> Item {
    int lo = 0, hi = S;                                              // largest s with first_tile[s] * f_tiles <= w and a non-empty segment
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (first_tile[mid] * f_tiles <= w) lo = mid; else hi = mid;
    }
    const MoeSegment sg = moe_segment(seg_off, n_routed, seg_rows, lo);
    const int tiles = first_tile[lo + 1] - first_tile[lo], r = w - first_tile[lo] * f_tiles;
    const int bn = ((sg.rows + tiles - 1) / tiles + 31) & ~31, t0 = (r % tiles) * bn;
    return {lo, (r / tiles) * TF, t0, bn, min(bn, sg.rows - t0), sg.row0};
  };

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      for (int w = first; w < num_items; w += step) {
        const Item it = item(w);
        const bool from_x = shared_from_x && it.seg >= n_routed;
        const CUtensorMap* tt = from_x ? &tmap_x : &tmap_a;
        const int tok0 = it.t0 + rank * (it.bn / 2) + (from_x ? 0 : static_cast<int>(it.row0));
        const int w0 = it.seg * N + it.f0 + rank * (TF / 2);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag, status, 740)) goto producer_done;
          uint8_t* sw = smem + stage * MP_STAGE_BYTES;
          if (rank == 0) mbar_expect_tx(&full_bar[stage], 2 * MP_STAGE_BYTES);
          const uint32_t bar = cluster_addr(&full_bar[stage], 0);
          if constexpr (GATED) {
            tma_load_5d_pair(sw, &tmap_b, bar, kb * MP_BK, 0, 0, it.f0 / 16 + rank * 4, it.seg);
          } else {
            tma_load_2d_pair(sw, &tmap_b, bar, kb * MP_BK, w0);
          }
          tma_load_2d_pair(sw + MP_HALF_BYTES, tt, bar, kb * MP_BK, tok0);    // 128 rows, of which bn / 2 are read
          if (++stage == MP_STAGES) { stage = 0; phase ^= 1u; }
        }
      }
    producer_done:;
    }
  } else if (warp == 1) {
    if (rank == 0) {
      const uint32_t s0 = smem_u32(smem);
      const uint64_t da0 = make_smem_desc_sw128(s0, 16, 1024), db0 = make_smem_desc_sw128(s0 + MP_HALF_BYTES, 16, 1024);
      int stage = 0, buf = 0;
      uint32_t phase = 0, acc_phase = 0;
      bool ok = true;
      for (int w = first; w < num_items && ok; w += step) {
        const Item it = item(w);
        const uint32_t idesc = make_idesc_bf16(256, it.bn, 0, 0);
        ok = __all_sync(0xffffffffu, mbar_wait(&tempty_bar[buf], acc_phase ^ 1u, abort_flag, status, 741));
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t tacc = tmem_base + static_cast<uint32_t>(buf * 256);
        for (int kb = 0; kb < num_kb; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, abort_flag, status, 742));
          if (!ok) break;
          tc_fence_after_sync();
          const uint64_t da = smem_desc_at(da0, stage * MP_STAGE_BYTES), db = smem_desc_at(db0, stage * MP_STAGE_BYTES);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < MP_BK / 16; ++k)
              umma_bf16_ss_pair(tacc, smem_desc_at(da, k * 32), smem_desc_at(db, k * 32), idesc, (kb | k) != 0 ? 1u : 0u);
            umma_commit_pair(&empty_bar[stage]);
            if (kb == num_kb - 1) umma_commit_pair(&tfull_bar[buf]);
          }
          __syncwarp();
          if (++stage == MP_STAGES) { stage = 0; phase ^= 1u; }
        }
        if (++buf == 2) { buf = 0; acc_phase ^= 1u; }
      }
    }
  } else {
    const int quad = warp & 3;          // TMEM lane quadrant this warp may read
    constexpr int WF = GATED ? 16 : 32; // features per warp
    constexpr int PIECES = WF / 8;      // 16-byte pieces of a row's features
    __nv_bfloat16* mine = reinterpret_cast<__nv_bfloat16*>(staging + (warp - 2) * 2048);     // [32 tokens][WF]
    int buf = 0;
    uint32_t acc_phase = 0;
    for (int w = first; w < num_items; w += step) {
      const Item it = item(w);
      const int f0 = it.f0 + rank * (TF / 2) + quad * WF;
      if (!__all_sync(0xffffffffu, mbar_wait(&tfull_bar[buf], acc_phase, abort_flag, status, 743))) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>(buf * 256);
      __nv_bfloat16* crow = C + static_cast<size_t>(it.row0 + it.t0) * ldc + f0;
      if (f0 < N) {                     // the same for the whole warp
#pragma unroll 1
        for (int c = 0; c * 32 < it.rows; ++c) {
          uint32_t v[32];
          tmem_ld_32x32(taddr + c * 32, v);
          tmem_wait_ld();
          if constexpr (GATED) {
            const bool up = lane >= 16;
#pragma unroll
            for (int j = 0; j < 32; j += 2) {              // lanes 0..15 finish token j, the others token j + 1
              const float other = __shfl_xor_sync(0xffffffffu, __uint_as_float(up ? v[j] : v[j + 1]), 16);
              const float own = __uint_as_float(up ? v[j + 1] : v[j]);
              mine[(j + (up ? 1 : 0)) * WF + (lane & 15)] = __float2bfloat16(up ? silu_mul(other, own) : silu_mul(own, other));
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) mine[j * WF + lane] = __float2bfloat16(ff_act<ACT>(__uint_as_float(v[j])));
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < PIECES; ++i) {
            const int e = i * 32 + lane, tok = e / PIECES, piece = e % PIECES;
            const uint4 o = *reinterpret_cast<const uint4*>(mine + tok * WF + piece * 8);
            if (c * 32 + tok < it.rows && f0 + piece * 8 < N)
              *reinterpret_cast<uint4*>(crow + static_cast<size_t>(c * 32 + tok) * ldc + piece * 8) = o;
          }
          __syncwarp();
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(&tempty_bar[buf], 0));
      if (++buf == 2) { buf = 0; acc_phase ^= 1u; }
    }
  }

  // Teardown. After an aborted wait there may be bulk copies in flight; give them time to land before either CTA exits.
  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
  }
}

int make_tmap_bf16_2d(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld, uint32_t box_inner, uint32_t box_outer);
int make_tmap_bf16_5d(CUtensorMap* out, const void* ptr, const uint64_t* dims, const uint64_t* strides, const uint32_t* box);

template <int ACT>
static int launch_moe_pair(const CUtensorMap& ta, const CUtensorMap& tx, const CUtensorMap& tb, void* C, const int* seg_off, int n_routed,
                           int n_shared, int seg_rows, int from_x, int N, int K, int ldc, int num_sms, int* status, cudaStream_t stream) {
  auto kern = moe_pair_kernel<ACT>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, MP_SMEM) != cudaSuccess) return -20;
    configured = true;
  }
  const cudaError_t e = launch_pdl(kern, dim3(num_sms / 2 * 2), dim3(MP_THREADS), static_cast<size_t>(MP_SMEM), stream, ta, tx, tb,
                                   static_cast<__nv_bfloat16*>(C), seg_off, n_routed, n_shared, seg_rows, from_x, N, K, ldc, status);
  return e == cudaSuccess ? 0 : -21;
}

// Arguments are those of rpeg_moe_gemm, checked there; gated: N a multiple of 16.
int moe_pair(const void* A, long long a_rows_total, const void* X, const void* B, void* C, const int* seg_off, int n_routed, int n_shared,
             int seg_rows, int N, int K, int lda, int ldx, int ldb, int ldc, int act, int num_sms, int* status, cudaStream_t stream) {
  const int S = n_routed + n_shared;
  CUtensorMap ta, tx, tb;
  int rc = make_tmap_bf16_2d(&ta, A, K, a_rows_total, lda, MP_BK, 128);
  if (rc) return rc;
  rc = X != nullptr ? make_tmap_bf16_2d(&tx, X, K, seg_rows, ldx, MP_BK, 128) : make_tmap_bf16_2d(&tx, A, K, a_rows_total, lda, MP_BK, 128);
  if (rc) return rc - 100;
  if (act == FF_SWIGLU) {
    const uint64_t row = ldb, dims[5] = {static_cast<uint64_t>(K), 16, 2, static_cast<uint64_t>(N / 16), static_cast<uint64_t>(S)};
    const uint64_t strides[4] = {row, N * row, 16 * row, 2 * N * row};
    const uint32_t box[5] = {MP_BK, 16, 2, 4, 1};
    rc = make_tmap_bf16_5d(&tb, B, dims, strides, box);
  } else {
    rc = make_tmap_bf16_2d(&tb, B, K, static_cast<uint64_t>(S) * N, ldb, MP_BK, 128);
  }
  if (rc) return rc - 200;
#define RPEG_MP(ACT_) \
  case ACT_: return launch_moe_pair<ACT_>(ta, tx, tb, C, seg_off, n_routed, n_shared, seg_rows, X != nullptr, N, K, ldc, num_sms, status, stream);
  switch (act) {
    RPEG_MP(FF_NONE)
    RPEG_MP(FF_GELU)
    RPEG_MP(FF_SWIGLU)
    RPEG_MP(FF_RELU2)
    default: return -4;
  }
#undef RPEG_MP
}

}  // namespace rpeg
