// Causal flash attention backward for sm_100a on packed variable-length sequences, head dim 128 (the forward pass: flash_attn.cu).
//
//   P = exp(Q K^T * scale - lse)     dP = dO V^T     dS = P * (dP - D),  D_q = rowsum(dO * O) from a small pre-pass
//   dV = P^T dO      dK = scale * dS^T Q      dQ = scale * dS K
//
// Two launches of one kernel. One keeps a 128-key tile and walks the query tiles at or below the diagonal (dK, dV; with grouped queries
// those of all heads that share the keys); the other keeps a 128-query tile and walks the key tiles up to the diagonal (dQ). Each sums
// what it owns in TMEM and writes it once, in bf16. Scores are formed twice that way, seven products per pair of tiles instead of five,
// but nothing is added up in memory: one kernel for all three has to add dQ to a [T, H * 128] fp32 buffer in memory, 64 KB per pair of
// tiles, which took longer than the two extra products and needed a clearing and a conversion pass around it.
//
// Both walk in the same way; "kept" tiles are A1, A2 and streamed ones B1, B2:
//                     A1  A2  B1  B2    scores S [128 x 64]   products
//   keys kept         K   V   Q   dO    S^T = K Q^T           dV += P^T dO,  dK += dS^T Q
//   queries kept      Q   dO  K   V     S   = Q K^T           dQ += dS K
// The streamed side is cut into sub-tiles of 64 rows. S and dP of a sub-tile take 128 TMEM columns; there are two such buffers, and each
// belongs to one of two groups of four warps (thread = kept row). While a group turns its S and dP into P and dS (bf16, in place: the
// next product reads them from TMEM), the tensor core forms the other buffer's scores and the products of the sub-tile before. 256 columns
// are left for the two accumulators. All loads are TMA, two stages of a streamed tile pair ahead.
//
// Bound by the tensor core (S, dP: 12 KB of shared memory per 128x64x16 step) and, close behind, by the 64 exponentials, conversions and
// TMEM transfers per thread and sub-tile. Against one kernel that ran one pair of tiles at a time and added dQ in memory, 32 heads:
// 8 x 2048 tokens 3.57 -> 1.25 ms (548 TFLOP/s); 16 x 1024 2.10 -> 0.89 ms; 2560, 2063, 1455, 848, 2241, 1633 tokens 2.42 -> 0.86 ms;
// 8 x 2048 with 8 KV heads 3.81 -> 1.14 ms.
#include "act_io.cuh"
#include "rpeg_kernels.h"

namespace rpeg {

int make_tmap_bf16_2d(CUtensorMap* out, const void* ptr, uint64_t inner, uint64_t outer, uint64_t ld,
                      uint32_t box_inner, uint32_t box_outer);

constexpr int FB_HD = 128, FB_T = 128, FB_SUB = 64, FB_STAGES = 2, FB_THREADS = 320;
constexpr int FB_TILE = FB_T * FB_HD * 2;                      // one tile: two 64-column 128B-swizzle atoms
constexpr int FB_ATOM = FB_TILE / 2, FB_SUB_BYTES = FB_SUB * 128;
constexpr int FB_VEC = 8 * 2 * 2 * FB_SUB * 4;                 // per warp, two turns: lse and D of a sub-tile's queries
constexpr int FB_SMEM = FB_TILE * (2 + 2 * FB_STAGES) + FB_VEC + 1024 + 256;

struct BwdArgs {
  const int* cu_seqlens;
  const float *lse, *dvec;        // [H, T]
  __nv_bfloat16* dqkv;
  int ld, T, H, Hkv, q_col0, k_col0, v_col0;
  float scale;
  int* status;
};

// D[h, t] = sum_d dO * O: 16 lanes per (token, head), 16-byte loads (two of 8 bytes where `o` is aligned to no more).
__global__ void __launch_bounds__(256)
attn_bwd_prep_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout, float* __restrict__ dvec, int T, int H) {
  const long long w = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 4;
  const bool live = w < static_cast<long long>(T) * H;
  const int lane = threadIdx.x & 15;
  float s = 0.f;
  if (live) {
    const size_t off = static_cast<size_t>(w) * FB_HD + lane * 8;
    const uint4 b = *reinterpret_cast<const uint4*>(dout + off);
    uint4 a;
    if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) {
      a = *reinterpret_cast<const uint4*>(o + off);
    } else {
      const uint2 lo = *reinterpret_cast<const uint2*>(o + off), hi = *reinterpret_cast<const uint2*>(o + off + 4);
      a = make_uint4(lo.x, lo.y, hi.x, hi.y);
    }
    const uint32_t *pa = reinterpret_cast<const uint32_t*>(&a), *pb = reinterpret_cast<const uint32_t*>(&b);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 x = unpack_bf16x2(pa[i]), y = unpack_bf16x2(pb[i]);
      s += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
  if (live && lane == 0) dvec[static_cast<size_t>(w % H) * T + w / H] = s;
}

template <bool KEEP_Q>
__global__ void __launch_bounds__(FB_THREADS, 1)
flash_attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_qkv, const __grid_constant__ CUtensorMap tmap_do, const BwdArgs p) {
  const int b = blockIdx.z, hy = blockIdx.y, G = p.H / p.Hkv;
  const int seq0 = p.cu_seqlens[b], L = p.cu_seqlens[b + 1] - seq0;
  const int tile = KEEP_Q ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x);   // most work first
  const int t0 = tile * FB_T;
  if (t0 >= L) return;
  const int all_sub = (L + FB_SUB - 1) / FB_SUB;
  const int sub0 = KEEP_Q ? 0 : 2 * tile;                        // first streamed sub-tile
  const int n_sub = (KEEP_Q ? min(all_sub, 2 * tile + 2) : all_sub) - sub0;
  const int heads = KEEP_Q ? 1 : G, head0 = KEEP_Q ? hy : hy * G, hk = KEEP_Q ? hy / G : hy;
  const int tiles = (n_sub + 1) / 2;                             // streamed tiles per head
  const int U = n_sub * heads;

  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* a1 = smem;
  uint8_t* a2 = a1 + FB_TILE;
  uint8_t* bst = a2 + FB_TILE;                                   // stage: B1, B2
  float* vec = reinterpret_cast<float*>(bst + 2 * FB_STAGES * FB_TILE);
  uint64_t* a_full = reinterpret_cast<uint64_t*>(vec + FB_VEC / 4);
  uint64_t* b_full = a_full + 1;                // [2]
  uint64_t* b_empty = b_full + FB_STAGES;       // [2] products that read the stage are done
  uint64_t* s_full = b_empty + FB_STAGES;       // [2] S and dP of the buffer are there
  uint64_t* p_full = s_full + 2;                // [2] P and dS are (4 warps)
  uint64_t* done = p_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(a_full, 1);
    mbar_init(done, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&b_full[s], 1);
      mbar_init(&b_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_full[s], 4);
    }
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
  const uint32_t tmem = *tmem_slot;
  constexpr uint32_t ACC2 = 256, ACC1 = 384;    // dV; dK or dQ

  if (warp == 0) {
    if (lane == 0) {
      tma_prefetch_desc(&tmap_qkv);
      tma_prefetch_desc(&tmap_do);
      auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int col, int row) {
        tma_load_2d(dst, map, bar, col, row);
        tma_load_2d(dst + FB_ATOM, map, bar, col + 64, row);
      };
      mbar_expect_tx(a_full, 2 * FB_TILE);
      load(a1, &tmap_qkv, a_full, KEEP_Q ? p.q_col0 + hy * FB_HD : p.k_col0 + hk * FB_HD, seq0 + t0);
      if (KEEP_Q) load(a2, &tmap_do, a_full, hy * FB_HD, seq0 + t0);
      else load(a2, &tmap_qkv, a_full, p.v_col0 + hk * FB_HD, seq0 + t0);
      int n = 0;
      bool ok = true;
      for (int h = 0; h < heads && ok; ++h) {
        for (int t = 0; t < tiles; ++t, ++n) {
          const int st = n & 1, row = seq0 + sub0 * FB_SUB + t * FB_T;
          if (!mbar_wait(&b_empty[st], (static_cast<uint32_t>(n >> 1) & 1u) ^ 1u, abort_flag, p.status, 600)) { ok = false; break; }
          uint8_t* dst = bst + st * 2 * FB_TILE;
          mbar_expect_tx(&b_full[st], 2 * FB_TILE);
          load(dst, &tmap_qkv, &b_full[st], KEEP_Q ? p.k_col0 + hk * FB_HD : p.q_col0 + (head0 + h) * FB_HD, row);
          if (KEEP_Q) load(dst + FB_TILE, &tmap_qkv, &b_full[st], p.v_col0 + hk * FB_HD, row);
          else load(dst + FB_TILE, &tmap_do, &b_full[st], (head0 + h) * FB_HD, row);
        }
      }
    }
  } else if (warp == 1) {
    // all lanes run the loop, one issues
    const bool leader = elect_one();
    constexpr uint32_t idesc_s = make_idesc_bf16(128, FB_SUB, 0, 0);       // both K-major
    constexpr uint32_t idesc_p = make_idesc_bf16(128, FB_HD, 0, 1);        // A in TMEM, B MN-major
    const uint64_t a1d = make_smem_desc_sw128(smem_u32(a1), 16, 1024), a2d = make_smem_desc_sw128(smem_u32(a2), 16, 1024);
    const uint64_t bk = make_smem_desc_sw128(smem_u32(bst), 16, 1024), bmn = make_smem_desc_sw128(smem_u32(bst), FB_ATOM, 1024);
    auto wait = [&](uint64_t* bar, uint32_t parity, int where) -> bool {
      return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, p.status, where));
    };
    int s_sub = 0, s_tile = 0;                   // of the next scores: sub-tile inside its head, streamed tile counted over all heads
    auto scores = [&](int u) -> bool {
      const int half = s_sub & 1, st = s_tile & 1;
      if (half == 0 && !wait(&b_full[st], static_cast<uint32_t>(s_tile >> 1) & 1u, 611)) return false;
      tc_fence_after_sync();
      const uint32_t ts = tmem + (u & 1) * 128u;
      const uint64_t b1d = smem_desc_at(bk, st * 2 * FB_TILE + half * FB_SUB_BYTES), b2d = smem_desc_at(b1d, FB_TILE);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t off = static_cast<uint32_t>((k >> 2) * FB_ATOM + (k & 3) * 32);
        if (leader) umma_bf16_ss(ts, smem_desc_at(a1d, off), smem_desc_at(b1d, off), idesc_s, k != 0 ? 1u : 0u);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t off = static_cast<uint32_t>((k >> 2) * FB_ATOM + (k & 3) * 32);
        if (leader) umma_bf16_ss(ts + FB_SUB, smem_desc_at(a2d, off), smem_desc_at(b2d, off), idesc_s, k != 0 ? 1u : 0u);
      }
      if (leader) umma_commit(&s_full[u & 1]);
      if (half == 1 || s_sub + 1 == n_sub) ++s_tile;
      if (++s_sub == n_sub) s_sub = 0;
      return true;
    };
    bool ok = wait(a_full, 0, 610) && scores(0);
    if (ok && U > 1) ok = scores(1);
    int sub = 0, n = 0;                          // of the products
    for (int u = 0; u < U && ok; ++u) {
      if (!wait(&p_full[u & 1], static_cast<uint32_t>(u >> 1) & 1u, 613)) break;
      tc_fence_after_sync();
      const int half = sub & 1, st = n & 1;
      const uint32_t ts = tmem + (u & 1) * 128u;
      const uint64_t b1d = smem_desc_at(bmn, st * 2 * FB_TILE + half * FB_SUB_BYTES), b2d = smem_desc_at(b1d, FB_TILE);
      if constexpr (!KEEP_Q) {
#pragma unroll
        for (int k = 0; k < FB_SUB / 16; ++k)    // 16 streamed rows: 8 columns of packed P, 2 KB of every atom of B2
          if (leader) umma_bf16_ts(tmem + ACC2, ts + k * 8, smem_desc_at(b2d, k * 2048), idesc_p, (u | k) != 0 ? 1u : 0u);
      }
#pragma unroll
      for (int k = 0; k < FB_SUB / 16; ++k)
        if (leader) umma_bf16_ts(tmem + ACC1, ts + FB_SUB + k * 8, smem_desc_at(b1d, k * 2048), idesc_p, (u | k) != 0 ? 1u : 0u);
      const bool last = half == 1 || sub + 1 == n_sub;
      if (leader && last) umma_commit(&b_empty[st]);
      if (last) ++n;
      if (++sub == n_sub) sub = 0;
      if (u + 2 < U) ok = scores(u + 2);         // into the buffer whose P and dS the products above read: they run in order
    }
    if (leader && ok) umma_commit(done);
  } else {
    const int quad = warp & 3, group = (warp - 2) >> 2, r = quad * 32 + lane;
    const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16);
    const uint32_t ts = lanes + group * 128u;
    const int mine = t0 + r;                     // the kept row, inside the sequence
    const float log2e = 1.4426950408889634f;
    const uint64_t scale2 = pack2(p.scale * log2e, p.scale * log2e);
    float* my_vec = vec + (warp - 2) * (4 * FB_SUB);   // two turns of { -lse, -D }
    // The exponent's and D's shifts: per kept row, or (keys kept) per streamed row, fetched one turn ahead. A query past the end of the
    // sequence gets -inf: its P is zero.
    auto shift_of = [&](int h, int qi) { return qi < L ? -log2e * p.lse[static_cast<size_t>(h) * p.T + seq0 + qi] : -INFINITY; };
    auto minus_d = [&](int h, int qi) { return qi < L ? -p.dvec[static_cast<size_t>(h) * p.T + seq0 + qi] : 0.f; };
    uint64_t row_l = 0, row_d = 0;
    float nl[2] = {0.f, 0.f}, nd[2] = {0.f, 0.f};
    int sub = group, h = head0;
    auto settle = [&]() { while (sub >= n_sub) { sub -= n_sub; ++h; } };
    auto fetch = [&]() {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int qi = (sub0 + sub) * FB_SUB + i * 32 + lane;
        nl[i] = shift_of(h, qi);
        nd[i] = minus_d(h, qi);
      }
    };
    if (KEEP_Q) {
      const float l = shift_of(hy, mine), d = minus_d(hy, mine);
      row_l = pack2(l, l);
      row_d = pack2(d, d);
    } else if (group < U) {
      settle();
      fetch();
    }
    bool ok = true;
    for (int u = group, turn = 0; u < U; u += 2, ++turn) {
      const int x0 = (sub0 + (KEEP_Q ? u : sub)) * FB_SUB;       // first streamed row
      float* v = my_vec + (turn & 1) * (2 * FB_SUB);
      if constexpr (!KEEP_Q) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { v[i * 32 + lane] = nl[i]; v[FB_SUB + i * 32 + lane] = nd[i]; }
        __syncwarp();
        sub += 2;
        if (u + 2 < U) { settle(); fetch(); }
      }
      if (!__all_sync(0xffffffffu, mbar_wait(&s_full[group], static_cast<uint32_t>(turn) & 1u, abort_flag, p.status, 620))) { ok = false; break; }
      tc_fence_after_sync();
      const bool mask = KEEP_Q ? x0 + FB_SUB - 1 > t0 : x0 < t0 + FB_T - 1;
      uint32_t s[2][16], d[2][16];
      tmem_ld_32x16(ts, s[0]);
      tmem_ld_32x16(ts + FB_SUB, d[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        tmem_wait_ld();
        if (c < 3) {
          tmem_ld_32x16(ts + (c + 1) * 16, s[(c + 1) & 1]);
          tmem_ld_32x16(ts + FB_SUB + (c + 1) * 16, d[(c + 1) & 1]);
        }
        uint32_t pp[8], dd[8];
#pragma unroll
        for (int i = 0; i < 8; i += 2) {
          uint64_t l2[2] = {row_l, row_l}, d2[2] = {row_d, row_d};
          if constexpr (!KEEP_Q) {
            const float4 a = load4(v + c * 16 + 2 * i), e = load4(v + FB_SUB + c * 16 + 2 * i);
            l2[0] = pack2(a.x, a.y); l2[1] = pack2(a.z, a.w);
            d2[0] = pack2(e.x, e.y); d2[1] = pack2(e.z, e.w);
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int j = 2 * (i + q);
            const float2 z = unpack2(fma2(pack2(__uint_as_float(s[c & 1][j]), __uint_as_float(s[c & 1][j + 1])), scale2, l2[q]));
            float p0 = exp2f(z.x), p1 = exp2f(z.y);
            if (mask) {
              const int x = x0 + c * 16 + j;
              if (KEEP_Q ? x > mine : x < mine) p0 = 0.f;
              if (KEEP_Q ? x + 1 > mine : x + 1 < mine) p1 = 0.f;
            }
            const float2 g = unpack2(mul2(pack2(p0, p1), add2(pack2(__uint_as_float(d[c & 1][j]), __uint_as_float(d[c & 1][j + 1])), d2[q])));
            pp[i + q] = pack_bf16x2(p0, p1);
            dd[i + q] = pack_bf16x2(g.x, g.y);
          }
        }
        // packed columns 8 c .. 8 c + 7: of S and dP, only chunks up to this one lie there
        if constexpr (!KEEP_Q) tmem_st_32x8(ts + c * 8, pp);
        tmem_st_32x8(ts + FB_SUB + c * 8, dd);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[group]);
    }
    if (ok && __all_sync(0xffffffffu, mbar_wait(done, 0, abort_flag, p.status, 621))) {
      tc_fence_after_sync();
      // keys kept: one group stores dV, the other dK; queries kept: half of dQ's columns each
      const bool scaled = KEEP_Q || group == 1;
      const uint32_t src = lanes + (scaled ? ACC1 : ACC2) + (KEEP_Q ? group * 64u : 0u);
      const int col = KEEP_Q ? p.q_col0 + hy * FB_HD + group * 64 : (group == 1 ? p.k_col0 : p.v_col0) + hk * FB_HD;
      const float sc = scaled ? p.scale : 1.f;
      __nv_bfloat16* dst = p.dqkv + static_cast<size_t>(seq0 + mine) * p.ld + col;
#pragma unroll 1
      for (int c = 0; c < (KEEP_Q ? 2 : 4); ++c) {
        uint32_t x[32];
        tmem_ld_32x32(src + c * 32, x);
        tmem_wait_ld();
        if (mine < L) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(x[i * 8 + 0]) * sc, __uint_as_float(x[i * 8 + 1]) * sc);
            o.y = pack_bf16x2(__uint_as_float(x[i * 8 + 2]) * sc, __uint_as_float(x[i * 8 + 3]) * sc);
            o.z = pack_bf16x2(__uint_as_float(x[i * 8 + 4]) * sc, __uint_as_float(x[i * 8 + 5]) * sc);
            o.w = pack_bf16x2(__uint_as_float(x[i * 8 + 6]) * sc, __uint_as_float(x[i * 8 + 7]) * sc);
            *reinterpret_cast<uint4*>(dst + c * 32 + i * 8) = o;
          }
        }
        __syncwarp();
      }
    }
  }

  __syncwarp();
  if (*abort_flag) __nanosleep(200000);
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, 512);
  }
}

template <bool KEEP_Q>
static int launch_bwd(const CUtensorMap& tm_qkv, const CUtensorMap& tm_do, const BwdArgs& p, int max_seqlen, int B, cudaStream_t stream) {
  auto kern = flash_attn_bwd_kernel<KEEP_Q>;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, FB_SMEM) != cudaSuccess) return -20;
    configured = true;
  }
  kern<<<dim3((max_seqlen + FB_T - 1) / FB_T, KEEP_Q ? p.H : p.Hkv, B), FB_THREADS, FB_SMEM, stream>>>(tm_qkv, tm_do, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -21;
}

}  // namespace rpeg

// qkv / out / lse are the forward's tensors; dout is [T, H * 128] bf16; dvec a scratch of [H, T] floats. dqkv ([T, ld_dqkv] bf16) receives
// dQ, dK, dV in the same column blocks as qkv.
extern "C" int rpeg_flash_attn_bwd(const void* qkv, int ld, int q_col0, int k_col0, int v_col0, const void* out,
                                   const void* dout, const float* lse, const int* cu_seqlens, int B,
                                   int max_seqlen, int T, int H, int Hkv, int hd, float scale, float* dvec,
                                   void* dqkv, int ld_dqkv, int* status, void* stream_v) {
  using namespace rpeg;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  if (hd != FB_HD || Hkv <= 0 || H % Hkv != 0) return -2;
  if ((ld | ld_dqkv | q_col0 | k_col0 | v_col0) & 7) return -3;
  if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dqkv)) & 15) return -1;
  if (B <= 0 || T <= 0 || max_seqlen <= 0) return 0;
  CUtensorMap tm_qkv, tm_do;
  int rc = make_tmap_bf16_2d(&tm_qkv, qkv, static_cast<uint64_t>(ld), static_cast<uint64_t>(T), static_cast<uint64_t>(ld), 64, FB_T);
  if (rc) return rc;
  rc = make_tmap_bf16_2d(&tm_do, dout, static_cast<uint64_t>(H) * FB_HD, static_cast<uint64_t>(T), static_cast<uint64_t>(H) * FB_HD, 64, FB_T);
  if (rc) return rc - 100;
  const long long rows = static_cast<long long>(T) * H;
  attn_bwd_prep_kernel<<<static_cast<unsigned>((rows * 16 + 255) / 256), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(out), static_cast<const __nv_bfloat16*>(dout), dvec, T, H);
  const BwdArgs p{cu_seqlens, lse, dvec, static_cast<__nv_bfloat16*>(dqkv), ld_dqkv, T, H, Hkv, q_col0, k_col0, v_col0, scale, status};
  rc = launch_bwd<false>(tm_qkv, tm_do, p, max_seqlen, B, stream);
  return rc ? rc : launch_bwd<true>(tm_qkv, tm_do, p, max_seqlen, B, stream);
}
