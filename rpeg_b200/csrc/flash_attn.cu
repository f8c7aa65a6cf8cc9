// Causal flash attention forward for sm_100a on packed variable-length sequences, head dim 128.
//
//   O = softmax(Q K^T * scale + causal) V      per (sequence, head)
//
// One CTA works on two neighbouring 128-row query tiles ("units") of one head over the same key tiles: while the softmax warps of one
// unit turn its scores into weights, the tensor cores multiply for the other one. (One tile per CTA, scores double buffered, was bound
// by its four softmax warps: 32 heads, 8 x 2048 tokens: 434 us, two units 331 us; 32 x 512: 256 and 175 us.)
//   S = Q K^T   : A = Q tile, B = K tile, both K-major in shared memory (two 64-column 128B-swizzle atoms each), 128 TMEM columns a unit;
//   O += P V    : A = P read directly from TMEM (bf16, written over the scores), B = V tile in shared memory, MN-major; the first 64
//                 keys are multiplied while the last ones are exponentiated.
// Roles: a TMA warp, an MMA warp (all lanes run the loop, one issues), four softmax warps per unit (thread = query row = TMEM lane, so row
// maximum and sum need no shuffles). The commit behind Q K^T of a unit's next tile also covers its P V before it.
// The running max is only refreshed when it grows by more than 8 (in log2 units); a stale max is exact after the final division by l, and
// it makes the O rescale (TMEM load, scale, store) rare.
//
// Q/K/V are column blocks of one packed [T, ld] bf16 activation (the fused QKV projection output);
// cu_seqlens[b] is the first row of sequence b. Outputs: O [T, H*128] bf16, LSE [H, T] fp32.
//
// Replaces the reference's attention: Megatron core attention with an explicit (1,1,s,s) causal
// mask (RPEG/runtime/workers/megatron_worker.py:457,691,1618) / F.scaled_dot_product_attention in
// calibrate.py:230-376.
#include "prefill_softmax.cuh"
#include "rpeg_kernels.h"

namespace rpeg {

constexpr int FA_BM = 128;   // query rows per unit
constexpr int FA_BN = 128;   // keys per tile
constexpr int FA_HD = 128;
constexpr int FA_THREADS = 320;
constexpr int FA_ATOM = 128 * 128;
constexpr int FA_TILE_BYTES = 2 * FA_ATOM;  // 32 KiB: one [128 x 128] bf16 tile (two 16 KiB atoms)
constexpr int FA_KV_STAGES = 2;
constexpr int FA_SMEM = FA_TILE_BYTES * (2 + 2 * FA_KV_STAGES) + 1024 + 256;

__global__ void __launch_bounds__(FA_THREADS, 1)
flash_attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const int* __restrict__ cu_seqlens,
                      __nv_bfloat16* __restrict__ out, float* __restrict__ lse_out, int T, int H, int Hkv,
                      int q_col0, int k_col0, int v_col0, float scale_log2, int* status) {
  const int b = blockIdx.z, h = blockIdx.y;
  const int seq0 = cu_seqlens[b];
  const int L = cu_seqlens[b + 1] - seq0;
  const int q_first = (gridDim.x - 1 - blockIdx.x) * 2 * FA_BM;       // late tiles have the most keys: first
  if (q_first >= L) return;
  const int hk = h / (H / Hkv);
  const bool has1 = q_first + FA_BM < L;
  // key tiles of a unit: up to the diagonal of its last row
  const int je0 = (min(L, q_first + FA_BM) + FA_BN - 1) / FA_BN, je1 = has1 ? (min(L, q_first + 2 * FA_BM) + FA_BN - 1) / FA_BN : 0;
  const int n_tiles = max(je0, je1);

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_sm = smem;                                               // [2]
  uint8_t* k_sm = smem + 2 * FA_TILE_BYTES;
  uint8_t* v_sm = k_sm + FA_KV_STAGES * FA_TILE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_sm + FA_KV_STAGES * FA_TILE_BYTES);
  uint64_t* q_full = bars;
  uint64_t* k_full = bars + 1;
  uint64_t* k_empty = k_full + FA_KV_STAGES;
  uint64_t* v_full = k_empty + FA_KV_STAGES;
  uint64_t* v_empty = v_full + FA_KV_STAGES;
  uint64_t* s_full = v_empty + FA_KV_STAGES;  // [2], per unit: S of its next tile is complete (and its P V before that)
  uint64_t* p_half = s_full + 2;              // [2], per unit: its weights for the first 64 keys are in place
  uint64_t* p_full = p_half + 2;              // [2], per unit: and for the others
  uint64_t* o_full = p_full + 2;              // [2], per unit: O is final
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 1);
    for (int s = 0; s < FA_KV_STAGES; ++s) {
      mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1);
      mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1);
    }
    for (int u = 0; u < 2; ++u) { mbar_init(&s_full[u], 1); mbar_init(&p_half[u], 4); mbar_init(&p_full[u], 4); mbar_init(&o_full[u], 1); }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_qkv);
      auto load = [&](uint8_t* dst, uint64_t* bar, int col, int row) {
        tma_load_2d(dst, &tmap_qkv, bar, col, row);
        tma_load_2d(dst + FA_ATOM, &tmap_qkv, bar, col + 64, row);
      };
      mbar_expect_tx(q_full, has1 ? 2 * FA_TILE_BYTES : FA_TILE_BYTES);
      load(q_sm, q_full, q_col0 + h * FA_HD, seq0 + q_first);
      if (has1) load(q_sm + FA_TILE_BYTES, q_full, q_col0 + h * FA_HD, seq0 + q_first + FA_BM);
      for (int j = 0; j < n_tiles; ++j) {
        const int st = j % FA_KV_STAGES;
        const uint32_t ph = static_cast<uint32_t>(j / FA_KV_STAGES) & 1u;
        if (!mbar_wait(&k_empty[st], ph ^ 1u, abort_flag, status, 500)) break;
        mbar_expect_tx(&k_full[st], FA_TILE_BYTES);
        load(k_sm + st * FA_TILE_BYTES, &k_full[st], k_col0 + hk * FA_HD, seq0 + j * FA_BN);
        if (!mbar_wait(&v_empty[st], ph ^ 1u, abort_flag, status, 501)) break;
        mbar_expect_tx(&v_full[st], FA_TILE_BYTES);
        load(v_sm + st * FA_TILE_BYTES, &v_full[st], v_col0 + hk * FA_HD, seq0 + j * FA_BN);
      }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    constexpr uint32_t idesc_qk = make_idesc_bf16(128, 128, 0, 0);
    constexpr uint32_t idesc_pv = make_idesc_bf16(128, 128, 0, 1);
    const uint64_t qd = make_smem_desc_sw128(smem_u32(q_sm), 16, 1024), kd = make_smem_desc_sw128(smem_u32(k_sm), 16, 1024);
    const uint64_t vd = make_smem_desc_sw128(smem_u32(v_sm), FA_ATOM, 1024);
    auto wait = [&](uint64_t* bar, uint32_t parity, int where) -> bool {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, status, where));
    };
    auto active = [&](int u, int j) -> bool { return j < (u ? je1 : je0); };
    // Q K^T of unit u over tile j; the tile's K buffer is free again once the last unit has used it
    auto issue_qk = [&](int u, int j) {
      const int st = j % FA_KV_STAGES;
      if (active(u, j)) {
        const uint64_t qa = smem_desc_at(qd, u * FA_TILE_BYTES), ka = smem_desc_at(kd, st * FA_TILE_BYTES);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = static_cast<uint32_t>((k >> 2) * FA_ATOM + (k & 3) * 32);
          if (leader) umma_bf16_ss(tmem_base + u * 128, smem_desc_at(qa, off), smem_desc_at(ka, off), idesc_qk, k != 0 ? 1u : 0u);
        }
        if (leader) umma_commit(&s_full[u]);
      }
      if (leader && u == 1) umma_commit(&k_empty[st]);
    };
    bool ok = wait(q_full, 0, 510) && wait(&k_full[0], 0, 511);
    if (ok) {
      tc_fence_after_sync();
      issue_qk(0, 0);
      issue_qk(1, 0);
      for (int j = 0; j < n_tiles && ok; ++j) {
        const int st = j % FA_KV_STAGES, st1 = (j + 1) % FA_KV_STAGES;
        if (!wait(&v_full[st], static_cast<uint32_t>(j / FA_KV_STAGES) & 1u, 514)) break;
        if (j + 1 < n_tiles && !wait(&k_full[st1], static_cast<uint32_t>((j + 1) / FA_KV_STAGES) & 1u, 512)) break;
        const uint64_t va = smem_desc_at(vd, st * FA_TILE_BYTES);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (active(u, j)) {
            const uint32_t tp = tmem_base + u * 128, to = tmem_base + 256 + u * 128;
#pragma unroll
            for (int half = 0; half < 2 && ok; ++half) {
              ok = wait(half ? &p_full[u] : &p_half[u], static_cast<uint32_t>(j) & 1u, 513 + half * 2);
              if (!ok) break;
              tc_fence_after_sync();
#pragma unroll
              for (int k = half * 4; k < half * 4 + 4; ++k)   // 16 keys per step: 8 packed TMEM columns of P, 16 rows (2 KiB) of the V tile
                if (leader) umma_bf16_ts(to, tp + k * 8, smem_desc_at(va, k * 2048), idesc_pv, (j | k) != 0 ? 1u : 0u);
            }
            if (!ok) break;
            if (leader && j + 1 == (u ? je1 : je0)) umma_commit(&o_full[u]);
          }
          if (leader && u == 1) umma_commit(&v_empty[st]);
          tc_fence_after_sync();
          if (j + 1 < n_tiles) issue_qk(u, j + 1);
        }
      }
    }
  } else {
    const int ui = (warp - 2) >> 2;
    const int q0 = q_first + ui * FA_BM, je = ui ? je1 : je0;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const int qi = q0 + r;  // position inside the sequence
    const bool row_valid = qi < L;
    const int lo = row_valid ? 0 : 1, hi = row_valid ? qi : 0;        // an absent row sees nothing
    const uint32_t ts = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + ui * 128;
    const uint32_t to = ts + 256;
    float m_ref = -INFINITY, l = 0.f;
    bool ok = true;
    for (int j = 0; j < je; ++j) {
      if (!__all_sync(0xffffffffu, mbar_wait(&s_full[ui], static_cast<uint32_t>(j) & 1u, abort_flag, status, 520))) { ok = false; break; }
      tc_fence_after_sync();
      const int k0 = j * FA_BN;
      WpRow<4> row;
      wp_load_row(ts, row);
      if (k0 + FA_BN - 1 > q0 || L - q0 < FA_BM) wp_mask_row(row, k0, lo, hi);
      const float tmax = wp_max_row(row) * scale_log2;        // scale > 0, so max commutes with the scaling
      if (j == 0) {
        m_ref = tmax;
      } else {
        const bool need = tmax > m_ref + WP_RESCALE;
        if (__any_sync(0xffffffffu, need)) {
          const float alpha = need ? (m_ref == -INFINITY ? 0.f : exp2f(m_ref - tmax)) : 1.f;
          if (need) { m_ref = tmax; l *= alpha; }
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t v[32];
            tmem_ld_32x32(to + c * 32, v);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * alpha);
            tmem_st_32x32(to + c * 32, v);
          }
        }
      }
      l += wp_exp_row_bf16(row, ts, scale_log2, m_ref == -INFINITY ? 0.f : m_ref, &p_half[ui]);
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[ui]);
    }
    if (ok && je > 0 && __all_sync(0xffffffffu, mbar_wait(&o_full[ui], 0, abort_flag, status, 522))) {
      tc_fence_after_sync();
      const float inv_l = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* orow = out + (static_cast<size_t>(seq0 + qi) * H + h) * FA_HD;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t v[32];
        tmem_ld_32x32(to + c * 32, v);
        tmem_wait_ld();
        if (row_valid) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(v[i * 8 + 0]) * inv_l, __uint_as_float(v[i * 8 + 1]) * inv_l);
            o.y = pack_bf16x2(__uint_as_float(v[i * 8 + 2]) * inv_l, __uint_as_float(v[i * 8 + 3]) * inv_l);
            o.z = pack_bf16x2(__uint_as_float(v[i * 8 + 4]) * inv_l, __uint_as_float(v[i * 8 + 5]) * inv_l);
            o.w = pack_bf16x2(__uint_as_float(v[i * 8 + 6]) * inv_l, __uint_as_float(v[i * 8 + 7]) * inv_l);
            *reinterpret_cast<uint4*>(orow + c * 32 + i * 8) = o;
          }
        }
      }
      if (row_valid && lse_out != nullptr)
        lse_out[static_cast<size_t>(h) * T + seq0 + qi] = ((m_ref == -INFINITY ? 0.f : m_ref) + log2f(l)) * 0.6931471805599453f;
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

int make_tmap_bf16_2d(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

}  // namespace rpeg

using namespace rpeg;

extern "C" int rpeg_flash_attn_fwd(const void* qkv, int ld, int q_col0, int k_col0, int v_col0,
                                   const int* cu_seqlens, int B, int max_seqlen, int T, int H, int Hkv, int hd,
                                   float scale, void* out, float* lse, int* status, void* stream_v) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (hd != FA_HD || H % Hkv != 0) return -2;
  if ((ld | q_col0 | k_col0 | v_col0) & 7) return -3;
  if (reinterpret_cast<uintptr_t>(qkv) & 15) return -1;
  if (B <= 0 || T <= 0 || max_seqlen <= 0) return 0;
  CUtensorMap tm;
  const int rc = make_tmap_bf16_2d(&tm, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(T),
                                   static_cast<uint64_t>(ld), 64, 128);
  if (rc) return rc;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(flash_attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FA_SMEM) != cudaSuccess)
      return -20;
    configured = true;
  }
  dim3 grid((max_seqlen + 2 * FA_BM - 1) / (2 * FA_BM), H, B);
  flash_attn_fwd_kernel<<<grid, FA_THREADS, FA_SMEM, stream>>>(tm, cu_seqlens, static_cast<__nv_bfloat16*>(out), lse,
                                                              T, H, Hkv, q_col0, k_col0, v_col0,
                                                              scale * 1.4426950408889634f, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}
