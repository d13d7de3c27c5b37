// Causal flash-attention backward for head_dim 128 on sm_100a (MHA and GQA).
//
// One CTA per (128-key tile, KV head or part of its query heads, sequence); it walks the 64-row query tiles of its query
// heads that attend to those keys.  Everything is computed with the keys in the TMEM lanes.  Per step five tcgen05 GEMMs:
//   S^T = K Q^T         dP^T = V dO^T                  (fp32 in TMEM, one key per lane, one query per column)
//   P^T = exp(S^T*scale - lse),  dS^T = P^T * (dP^T - D)   (softmax warps; bf16 back into TMEM, dS^T also into shared memory)
//   dV += P^T dO        dK += dS^T Q                   (A operand from TMEM; accumulated in TMEM over the whole walk)
//   dQ^T = K^T dS^T     -> TMEM -> shared memory -> added to a global fp32 dQ accumulator by TMA reduce-add
// Roles:
//   warps 0-3, 4-7   softmax of the even / odd steps, one thread per key
//   warps 8-11       dQ^T: out of TMEM, transposed through shared memory, one TMA reduce-add per warp and step
//   warp 12          TMA producer: K and V once, then Q and dO through a ring of three stages
//   warp 13          MMA issuer
//   warp 14          the query rows' statistics for the ring, read one step ahead
// TMEM (512 columns): dV, dK (128 each) and two sets (even / odd steps) of [S^T | dP^T], 64 columns each: P^T and dS^T
// (bf16, 16 + 16 columns per 32 queries) replace S^T once it has been read, dQ^T replaces dP^T.  So the softmax of one step runs under
// the MMAs of its neighbours.  Bound: about 1700 cycles of MMA per step (S^T, dP^T and dQ^T with N = 64 are limited by the
// 128 bytes per cycle that shared memory delivers: 48 instead of 32 cycles per instruction).
// D = rowsum(dO * O) comes from a small pre-pass; scale and bf16 of dQ are applied by a post-pass, of dK at the end.
#include <stdio.h>

#include "common.cuh"
#include "yafsdp_b200.h"

YF_TU_STATUS()

namespace {

constexpr int HD = 128;
constexpr int BQ = 64;    // query rows per step
constexpr int BKV = 128;  // keys per CTA
constexpr int ATOM = 16384;        // [128 rows x 64 bf16], 128-byte swizzle
constexpr int TILE = 2 * ATOM;     // K or V: [128 x 128] bf16
constexpr int QATOM = 8192;        // [64 rows x 64 bf16]
constexpr int QTILE = 2 * QATOM;   // Q or dO of a step: [64 x 128] bf16
constexpr int STAGES = 3;          // ring of Q, dO and statistics
constexpr int BWD_THREADS = 480;
constexpr int DS_BYTES = ATOM;     // dS^T of a step: [128 keys x 64 queries] bf16
constexpr int DQ_BYTES = BQ * HD * 4;
constexpr int STAT_FLOATS = 2 * BQ;  // per stage: -lse * log2(e), D
constexpr int BWD_SMEM = 1024 + 2 * TILE + STAGES * 2 * QTILE + 2 * DS_BYTES + DQ_BYTES + STAGES * STAT_FLOATS * 4 + 256;
static_assert(BWD_SMEM <= 232448, "shared memory of one CTA");

struct BwdArgs {
  const float* lse;    // [B, Hq, S]
  const float* delta;  // [B, Hq, S]
  __nv_bfloat16* dk;   // rows dkv_stride apart, head hk at columns hk*128
  __nv_bfloat16* dv;
  float4* dkv_parts;   // head_parts > 1: every part's own fp32 sums (part_tile), dK without scale; else null
  const float* rope;   // optional [S, 64, 2] (cos, sin): dK goes back through the rotation of K (head dims j and j + 64)
  long long dkv_stride;
  int S, B, Hq, Hkv;
  int head_group;      // order of the CTAs (head_group_order)
  int head_parts;      // CTAs that share a key tile of a KV head, each with a part of its query heads
  float scale, scale_log2;
  int causal;
};

YF_DEVINL void tma_reduce_add_3d(const CUtensorMap* m, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// Where a CTA that shares its key tile leaves dK (is_v = 0) and dV: [head_parts][B][key tiles][Hkv][2] blocks of 32 groups of four head
// dims x 128 keys, so that a warp, one key per lane, stores 512 contiguous bytes at a time (rows of 128 dims: 16 bytes in each of
// 32 lines).
constexpr int PART_TILE = BKV * HD / 4;  // float4s of a block
__host__ __device__ inline long long part_tile(int part, int B, int b, int n_kt, int jt, int Hkv, int hk, int is_v) {
  return (((((long long)part * B + b) * n_kt + jt) * Hkv + hk) * 2 + is_v) * PART_TILE;
}

// Order of the CTAs: heads are taken in groups, within a group key tile by key tile with the heads fastest, so that all heads'
// long walks start first.  One group holds all heads unless the dQ accumulator outgrows the L2 and there are heads for three
// groups; then a group has two CTAs per SM, whose sums stay in the L2.  It pays for many sequences or long ones: 8 x 2048 tokens x 32
// heads 1449 us in one group, 1247 in groups of 19; 2 x 8192 x 32 3516 / 3438 in groups of five; 2 x 2304 x 32 393 / 380; 2 x 4096 x
// 32 971 / 995 in groups of ten; 1 x 4096 x 64 984 / 1013.  1 x 8192 x 32/8 stays whole: 1543 us, 1572 in two groups.
YF_DEVINL void head_group_order(int cta, int n_pos, int n_heads, int group, int& pos, int& head) {
  const int per_group = n_pos * group;
  const int g = cta / per_group;
  const int r = cta - g * per_group;
  const int size = min(group, n_heads - g * group);
  pos = r / size;
  head = g * group + r - pos * size;
}
int head_group_size(int n_pos, int n_heads, long long accum_bytes, int n_sms) {
  const int group = (2 * n_sms + n_pos - 1) / n_pos;
  return accum_bytes <= (64ll << 20) || group >= n_heads / 3 ? n_heads : group;
}

// SHARED: head_parts > 1 (an instantiation of its own: the parts' addresses cost the other one registers it does not have)
template <bool SHARED>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                const __grid_constant__ CUtensorMap tma_v, const __grid_constant__ CUtensorMap tma_do,
                const __grid_constant__ CUtensorMap tma_dq, BwdArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sK = smem;
  uint8_t* sV = sK + TILE;
  uint8_t* sRing = sV + TILE;                      // stage s: Q at sRing + s * 2 * QTILE, dO at + QTILE
  uint8_t* sdS = sRing + STAGES * 2 * QTILE;       // even / odd steps
  uint8_t* sdQ = sdS + 2 * DS_BYTES;               // warp w of the dQ warps: [64 queries x 32 dims] fp32 at w * 8192
  float* sStat = reinterpret_cast<float*>(sdQ + DQ_BYTES);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sStat + STAGES * STAT_FLOATS);
  uint64_t* kv_full = bars;
  uint64_t* q_full = bars + 1;              // [STAGES] TMA bytes + the statistics
  uint64_t* q_empty = q_full + STAGES;      // [STAGES]
  uint64_t* sdp_full = q_empty + STAGES;    // [2] even / odd steps, as all that follow
  uint64_t* pds_ready = sdp_full + 2;
  uint64_t* dq_full = pds_ready + 2;
  uint64_t* vk_done = dq_full + 2;
  uint64_t* dq_read = vk_done + 2;
  uint64_t* all_done = dq_read + 2;         // every MMA of the walk (waiting two phases ahead on vk_done would not do)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(all_done + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  int jt, bh;  // key tile (under the causal mask the first ones have the longest walks), (sequence, KV head, part)
  const int head_parts = SHARED ? args.head_parts : 1;
  head_group_order((int)blockIdx.x, (args.S + BKV - 1) / BKV, args.B * args.Hkv * head_parts, args.head_group, jt, bh);
  const int part = bh % head_parts, hk = (bh / head_parts) % args.Hkv, b = bh / (head_parts * args.Hkv);
  const int heads = args.Hq / args.Hkv / head_parts;  // query heads of this CTA
  const int h0 = hk * (args.Hq / args.Hkv) + part * heads;
  const int kv0 = jt * BKV;
  const int i_start = args.causal ? kv0 / BQ : 0;          // first query tile
  const int per_head = (args.S + BQ - 1) / BQ - i_start;   // at least one: the tile that holds these keys' own rows
  const int n_it = per_head * heads;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_q);
    tma_prefetch_desc(&tma_k);
    tma_prefetch_desc(&tma_v);
    tma_prefetch_desc(&tma_do);
    tma_prefetch_desc(&tma_dq);
    mbar_init(kv_full, 1);
    mbar_init(all_done, 1);
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&q_full[i], 2);
      mbar_init(&q_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&sdp_full[i], 1);
      mbar_init(&pds_ready[i], 4);
      mbar_init(&dq_full[i], 1);
      mbar_init(&vk_done[i], 1);
      mbar_init(&dq_read[i], 4);
    }
    mbar_fence_init();
  }
  if (warp == 13) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t tdV = tmem_base + 256, tdK = tmem_base + 384;  // set p of S^T | dP^T: tmem_base + 128 p, + 64

  if (warp == 12) {
    if (elect_one()) {
      mbar_expect_tx(kv_full, 2 * TILE);
      tma_load_3d(sK, &tma_k, kv_full, hk * HD, kv0, b);
      tma_load_3d(sK + ATOM, &tma_k, kv_full, hk * HD + 64, kv0, b);
      tma_load_3d(sV, &tma_v, kv_full, hk * HD, kv0, b);
      tma_load_3d(sV + ATOM, &tma_v, kv_full, hk * HD + 64, kv0, b);
      int h = h0, i = 0;
      for (int it = 0, st = 0, ph = 1; it < n_it; ++it) {
        if (!mbar_wait(&q_empty[st], ph, 200)) break;
        const int q0 = (i_start + i) * BQ;
        uint8_t* sQ = sRing + st * 2 * QTILE;
        uint8_t* sdO = sQ + QTILE;
        mbar_expect_tx(&q_full[st], 2 * QTILE);
        tma_load_3d(sQ, &tma_q, &q_full[st], h * HD, q0, b);
        tma_load_3d(sQ + QATOM, &tma_q, &q_full[st], h * HD + 64, q0, b);
        tma_load_3d(sdO, &tma_do, &q_full[st], h * HD, q0, b);
        tma_load_3d(sdO + QATOM, &tma_do, &q_full[st], h * HD + 64, q0, b);
        if (++i == per_head) { i = 0; ++h; }
        if (++st == STAGES) { st = 0; ph ^= 1; }
      }
    }
  } else if (warp == 14) {
    // statistics of a step's 64 query rows, read one step ahead; rows past the end of the sequence: a probability of zero
    int h = h0, i = 0;
    float nl[2], dl[2];
    auto fetch = [&]() {
      const int q0 = (i_start + i) * BQ;
      const long long at = ((long long)b * args.Hq + h) * args.S + q0;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = lane + 32 * e;
        const bool ok = q0 + r < args.S;
        nl[e] = ok ? args.lse[at + r] * -1.4426950408889634f : -INFINITY;
        dl[e] = ok ? args.delta[at + r] : 0.f;
      }
    };
    fetch();
    for (int it = 0, st = 0, ph = 1; it < n_it; ++it) {
      if (!__all_sync(0xffffffffu, mbar_wait(&q_empty[st], ph, 201))) break;
      float* stat = sStat + st * STAT_FLOATS;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        stat[lane + 32 * e] = nl[e];
        stat[BQ + lane + 32 * e] = dl[e];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&q_full[st]);
      if (++i == per_head) { i = 0; ++h; }
      if (it + 1 < n_it) fetch();
      if (++st == STAGES) { st = 0; ph ^= 1; }
    }
  } else if (warp == 13) {
    if (elect_one()) {
      const uint32_t id_s = umma_idesc_bf16(128, BQ, 0, 0);    // S^T, dP^T: both operands K-major (K = head dim)
      const uint32_t id_g = umma_idesc_bf16(128, HD, 0, 1);    // dV, dK: A from TMEM (K = queries), dO / Q MN-major
      const uint32_t id_q = umma_idesc_bf16(128, BQ, 1, 1);    // dQ^T: K tile MN-major (M = head dim), dS^T MN-major
      const uint64_t kK = umma_smem_desc_sw128(smem_u32(sK), 0, 1024), kV = umma_smem_desc_sw128(smem_u32(sV), 0, 1024);
      const uint64_t mK = umma_smem_desc_sw128(smem_u32(sK), ATOM, 1024);
      const uint64_t kQ = umma_smem_desc_sw128(smem_u32(sRing), 0, 1024), mQ = umma_smem_desc_sw128(smem_u32(sRing), QATOM, 1024);
      const uint64_t mS = umma_smem_desc_sw128(smem_u32(sdS), ATOM, 1024);
      // descriptor addresses advance in units of 16 bytes
      int st_s = 0, ph_s = 0;  // ring position of the next S^T, dP^T
      // S^T and dP^T of step `it` into their set: S^T once dV and dK of step it - 2 have read P^T and dS^T there, dP^T once
      // the dQ warps have read dQ^T
      auto issue_sdp = [&](int it) -> bool {
        const int p = it & 1, par = ((it >> 1) & 1) ^ 1;  // parity of step it - 2
        if (!mbar_wait(&q_full[st_s], ph_s, 211)) return false;
        if (it >= 2 && !mbar_wait(&vk_done[p], par, 212)) return false;
        tc_fence_after();
        const uint64_t q = kQ + st_s * (2 * QTILE >> 4);
        const uint32_t t = tmem_base + p * 128;
#pragma unroll
        for (int e = 0; e < HD / 16; ++e)
          tc_mma_bf16(t, kK + (((e >> 2) * ATOM + (e & 3) * 32) >> 4), q + (((e >> 2) * QATOM + (e & 3) * 32) >> 4), id_s, e != 0);
        if (it >= 2 && !mbar_wait(&dq_read[p], par, 213)) return false;
        tc_fence_after();
#pragma unroll
        for (int e = 0; e < HD / 16; ++e)
          tc_mma_bf16(t + 64, kV + (((e >> 2) * ATOM + (e & 3) * 32) >> 4), q + ((QTILE + (e >> 2) * QATOM + (e & 3) * 32) >> 4), id_s,
                      e != 0);
        tc_commit(&sdp_full[p]);
        if (++st_s == STAGES) { st_s = 0; ph_s ^= 1; }
        return true;
      };
      bool alive = mbar_wait(kv_full, 0, 210) && issue_sdp(0) && (n_it < 2 || issue_sdp(1));
      int st = 0;
      for (int it = 0; it < n_it && alive; ++it) {
        const int p = it & 1;
        if (!mbar_wait(&pds_ready[p], (it >> 1) & 1, 214)) break;
        tc_fence_after();
        const uint32_t t = tmem_base + p * 128;
#pragma unroll
        for (int e = 0; e < BKV / 16; ++e)  // dQ^T first: the dQ warps fetch it under dV and dK
          tc_mma_bf16(t + 64, mK + e * (2048 >> 4), mS + ((p * DS_BYTES + e * 2048) >> 4), id_q, e != 0);
        tc_commit(&dq_full[p]);
        const uint64_t q = mQ + st * (2 * QTILE >> 4);
#pragma unroll
        for (int e = 0; e < BQ / 16; ++e)  // 16 queries: 8 TMEM columns of P^T, 16 rows of dO
          tc_mma_bf16_ts(tdV, t + (e >> 1) * 32 + (e & 1) * 8, q + ((QTILE + e * 2048) >> 4), id_g, (it | e) != 0);
#pragma unroll
        for (int e = 0; e < BQ / 16; ++e)
          tc_mma_bf16_ts(tdK, t + (e >> 1) * 32 + 16 + (e & 1) * 8, q + (e * 2048 >> 4), id_g, (it | e) != 0);
        tc_commit(&vk_done[p]);
        tc_commit(&q_empty[st]);
        if (++st == STAGES) st = 0;
        if (it + 2 < n_it) alive = issue_sdp(it + 2);
        if (it + 1 == n_it) tc_commit(all_done);
      }
    }
  } else if (warp < 8) {
    const int p = warp >> 2;                  // even or odd steps
    const int row = (warp & 3) * 32 + lane;   // key inside the tile == TMEM lane
    const uint32_t t = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + p * 128;
    const int key = kv0 + row;
    const float sl2 = args.scale_log2;
    uint8_t* ds_row = sdS + p * DS_BYTES + row * 128;
    bool alive = true;
    int st = p, ph = 0, i = p % per_head;     // ring stage and its parity, query tile of step p
    for (int it = p; it < n_it; it += 2) {
      const int q0 = (i_start + i) * BQ;
      // a bounded wait that runs out ends the warp's work (the lanes decide together: TMEM accesses are warp-wide)
      if (!__all_sync(0xffffffffu, mbar_wait(&q_full[st], ph, 220) && mbar_wait(&sdp_full[p], (it >> 1) & 1, 221))) { alive = false; break; }
      tc_fence_after();
      const float4* stat = reinterpret_cast<const float4*>(sStat + st * STAT_FLOATS);
      // queries [0, hidden) of the tile do not see this key: those in front of it, all when the key is past the end
      const int hidden = key >= args.S ? BQ : (args.causal ? key - q0 : 0);
      const bool any_hidden = __any_sync(0xffffffffu, hidden > 0);
      // 32 queries at a time: all but a few words (28 bytes, 52 with shared key tiles) stay in registers; a spill goes to the L2, as
      // shared memory leaves no L1
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t s[32], dp[32], pk[16], dk[16];
        tmem_ld32(t + c * 32, s);
        tmem_ld32(t + 64 + c * 32, dp);
        tmem_ld_wait();
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const float4 nl = stat[c * 8 + v], dl = stat[BQ / 4 + c * 8 + v];
          float x[4] = {fast_exp2(fmaf(__uint_as_float(s[4 * v + 0]), sl2, nl.x)), fast_exp2(fmaf(__uint_as_float(s[4 * v + 1]), sl2, nl.y)),
                        fast_exp2(fmaf(__uint_as_float(s[4 * v + 2]), sl2, nl.z)), fast_exp2(fmaf(__uint_as_float(s[4 * v + 3]), sl2, nl.w))};
          if (any_hidden) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (c * 32 + 4 * v + e < hidden) x[e] = 0.f;
          }
          pk[2 * v] = pack_bf16x2(x[0], x[1]);
          pk[2 * v + 1] = pack_bf16x2(x[2], x[3]);
          dk[2 * v] = pack_bf16x2(x[0] * (__uint_as_float(dp[4 * v + 0]) - dl.x), x[1] * (__uint_as_float(dp[4 * v + 1]) - dl.y));
          dk[2 * v + 1] = pack_bf16x2(x[2] * (__uint_as_float(dp[4 * v + 2]) - dl.z), x[3] * (__uint_as_float(dp[4 * v + 3]) - dl.w));
        }
        // over the half of S^T that has been read: P^T, then dS^T
        tmem_st16(t + c * 32, pk);
        tmem_st16(t + c * 32 + 16, dk);
#pragma unroll
        for (int v = 0; v < 4; ++v)
          *reinterpret_cast<uint4*>(ds_row + (((c * 4 + v) ^ (row & 7)) << 4)) = make_uint4(dk[4 * v], dk[4 * v + 1], dk[4 * v + 2], dk[4 * v + 3]);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pds_ready[p]);
      i += 2;
      while (i >= per_head) i -= per_head;
      st += 2;
      if (st >= STAGES) { st -= STAGES; ph ^= 1; }
    }
    // the results: the even steps' warps write dV, the odd steps' warps dK (TMEM lane == key)
    if (alive && __all_sync(0xffffffffu, mbar_wait(all_done, 0, 222))) {
      tc_fence_after();
      const uint32_t src = (p == 0 ? tdV : tdK) + ((uint32_t)((warp & 3) * 32) << 16);
      const float f = p == 0 ? 1.f : args.scale;
      const long long token = (long long)b * args.S + key;
      if (!SHARED && p == 1 && args.rope != nullptr) {
        const float4* cs = reinterpret_cast<const float4*>(args.rope + (long long)min(key, args.S - 1) * HD);  // two dims each
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {  // 16 dims and their partners
          uint32_t a[16], z[16];
          tmem_ld16(src + c * 16, a);
          tmem_ld16(src + 64 + c * 16, z);
          tmem_ld_wait();
          if (key < args.S) {
            uint32_t lo[8], hi[8];
#pragma unroll
            for (int v = 0; v < 8; ++v) {
              const float4 t4 = __ldg(cs + c * 8 + v);
              const float a0 = __uint_as_float(a[2 * v]), a1 = __uint_as_float(a[2 * v + 1]), z0 = __uint_as_float(z[2 * v]), z1 = __uint_as_float(z[2 * v + 1]);
              lo[v] = pack_bf16x2((a0 * t4.x + z0 * t4.y) * f, (a1 * t4.z + z1 * t4.w) * f);
              hi[v] = pack_bf16x2((z0 * t4.x - a0 * t4.y) * f, (z1 * t4.z - a1 * t4.w) * f);
            }
            uint4* dst = reinterpret_cast<uint4*>(args.dk + token * args.dkv_stride + hk * HD + c * 16);
            dst[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            dst[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
            dst[8] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            dst[9] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
          }
        }
      } else
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld32(src + c * 32, r);
        tmem_ld_wait();
        if (key < args.S) {
          if (SHARED) {
            float4* dst = args.dkv_parts + part_tile(part, args.B, b, (args.S + BKV - 1) / BKV, jt, args.Hkv, hk, p == 0 ? 1 : 0) + row;
#pragma unroll
            for (int v = 0; v < 8; ++v)
              dst[(c * 8 + v) * BKV] = make_float4(__uint_as_float(r[4 * v]), __uint_as_float(r[4 * v + 1]), __uint_as_float(r[4 * v + 2]),
                                                   __uint_as_float(r[4 * v + 3]));
          } else {
            uint4* dst = reinterpret_cast<uint4*>((p == 0 ? args.dv : args.dk) + token * args.dkv_stride + hk * HD + c * 32);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              uint4 w;
              w.x = pack_bf16x2(__uint_as_float(r[8 * v + 0]) * f, __uint_as_float(r[8 * v + 1]) * f);
              w.y = pack_bf16x2(__uint_as_float(r[8 * v + 2]) * f, __uint_as_float(r[8 * v + 3]) * f);
              w.z = pack_bf16x2(__uint_as_float(r[8 * v + 4]) * f, __uint_as_float(r[8 * v + 5]) * f);
              w.w = pack_bf16x2(__uint_as_float(r[8 * v + 6]) * f, __uint_as_float(r[8 * v + 7]) * f);
              dst[v] = w;
            }
          }
        }
      }
    }
    tc_fence_before();
  } else if (warp < 12) {
    const int w = warp & 3;                   // head dims [32 w, +32) == TMEM lanes
    float* stg = reinterpret_cast<float*>(sdQ) + w * (BQ * 32);
    int h = h0, i = 0;
    for (int it = 0; it < n_it; ++it) {
      const int p = it & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(&dq_full[p], (it >> 1) & 1, 230))) break;
      tc_fence_after();
      const uint32_t t = tmem_base + ((uint32_t)(w * 32) << 16) + p * 128 + 64;
      uint32_t r[2][32];
      tmem_ld32(t, r[0]);
      tmem_ld32(t + 32, r[1]);
      tmem_ld_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&dq_read[p]);
        tma_store_wait_read0();  // the reduce of the step before has finished reading the block
      }
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 32; ++e) stg[(c * 32 + e) * 32 + lane] = __uint_as_float(r[c][e]);
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        // rows past the end of the sequence are clipped by the tensor map
        tma_reduce_add_3d(&tma_dq, stg, h * HD + w * 32, (i_start + i) * BQ, b);
        tma_store_commit();
      }
      if (++i == per_head) { i = 0; ++h; }
    }
    if (lane == 0) tma_store_wait0();  // this warp's reduce-adds have completed
    tc_fence_before();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// delta[b,h,s] = sum_d dO * O, and the fp32 dQ accumulator of the same (token, head) cleared on the way (the main kernel
// adds into it): sixteen lanes per (token, head), one 16-byte load of O and of dO and two 16-byte stores of zeros per lane.
__global__ void __launch_bounds__(256) attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ d_o,
                                                         float* __restrict__ delta, float* __restrict__ dq_zero, int B, int S, int Hq,
                                                         long long o_stride, long long do_stride) {
  const long long total = (long long)B * S * Hq;
  const int sub = threadIdx.x & 15;
  const unsigned half_mask = 0xffffu << (threadIdx.x & 16);  // the two halves of a warp may leave the loop at different times
  for (long long w = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 4; w < total;
       w += ((long long)gridDim.x * blockDim.x) >> 4) {
    const int h = (int)(w % Hq);
    const long long t = w / Hq;
    const uint4 a = *reinterpret_cast<const uint4*>(o + t * o_stride + h * HD + sub * 8);
    const uint4 g = *reinterpret_cast<const uint4*>(d_o + t * do_stride + h * HD + sub * 8);
    if (dq_zero != nullptr) {
      float4* z = reinterpret_cast<float4*>(dq_zero + (t * Hq + h) * HD + sub * 8);
      z[0] = make_float4(0.f, 0.f, 0.f, 0.f);
      z[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const float2 a0 = unpack_bf16x2(a.x), a1 = unpack_bf16x2(a.y), a2 = unpack_bf16x2(a.z), a3 = unpack_bf16x2(a.w);
    const float2 g0 = unpack_bf16x2(g.x), g1 = unpack_bf16x2(g.y), g2 = unpack_bf16x2(g.z), g3 = unpack_bf16x2(g.w);
    float s = a0.x * g0.x + a0.y * g0.y + a1.x * g1.x + a1.y * g1.y + a2.x * g2.x + a2.y * g2.y + a3.x * g3.x + a3.y * g3.y;
#pragma unroll
    for (int m = 8; m >= 1; m >>= 1) s += __shfl_xor_sync(half_mask, s, m);
    if (sub == 0) {
      const long long bb = t / S, ss = t % S;
      delta[(bb * Hq + h) * S + ss] = s;
    }
  }
}

// dst, dst + 64 (bf16) = f * (a, z): eight head dims and their partners 64 further on.  With `cs` (cos, sin of the eight dims) they
// go back through the rotation on the way.
YF_DEVINL void store_gradient(__nv_bfloat16* dst, float (&a)[8], float (&z)[8], const float4* cs, float f) {
  if (cs != nullptr) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 c = __ldg(cs + j);
      const float a0 = a[2 * j], a1 = a[2 * j + 1];
      a[2 * j] = a0 * c.x + z[2 * j] * c.y;
      a[2 * j + 1] = a1 * c.z + z[2 * j + 1] * c.w;
      z[2 * j] = z[2 * j] * c.x - a0 * c.y;
      z[2 * j + 1] = z[2 * j + 1] * c.z - a1 * c.w;
    }
  }
  uint4 w;
  w.x = pack_bf16x2(a[0] * f, a[1] * f); w.y = pack_bf16x2(a[2] * f, a[3] * f);
  w.z = pack_bf16x2(a[4] * f, a[5] * f); w.w = pack_bf16x2(a[6] * f, a[7] * f);
  *reinterpret_cast<uint4*>(dst) = w;
  w.x = pack_bf16x2(z[0] * f, z[1] * f); w.y = pack_bf16x2(z[2] * f, z[3] * f);
  w.z = pack_bf16x2(z[4] * f, z[5] * f); w.w = pack_bf16x2(z[6] * f, z[7] * f);
  *reinterpret_cast<uint4*>(dst + 64) = w;
}
YF_DEVINL const float4* rope_at(const float* rope, int pos, int dim) {
  return rope == nullptr ? nullptr : reinterpret_cast<const float4*>(rope + ((long long)pos * 64 + dim) * 2);
}

// dq (bf16, strided rows) = scale * dq_accum (fp32, dense rows of 128 Hq); with dkv_parts also dk = scale * the sum of the parts' dK and
// dv = that of their dV, in the order of the parts.  `rope` ([S, 64, 2]: cos, sin): dq and dk go back through the rotation.
__global__ void __launch_bounds__(256) attn_convert_kernel(const float* __restrict__ dq_acc, const float4* __restrict__ dkv_parts, int parts, const float* __restrict__ rope,
                                    __nv_bfloat16* __restrict__ dq, __nv_bfloat16* __restrict__ dk, __nv_bfloat16* __restrict__ dv, int B,
                                    int S, int Hq, int Hkv, long long dq_stride, long long dkv_stride, float scale) {
  const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
  const long long n_dq = (long long)B * S * Hq * 8;
  const int n_kt = (S + BKV - 1) / BKV;
  const long long blocks = dkv_parts == nullptr ? 0 : (long long)B * n_kt * Hkv * 2;  // of a part
  const long long total = n_dq + blocks * (BKV * 8);
  for (long long i = first; i < total; i += step) {
    float a[8], z[8];
    if (i < n_dq) {
      const long long t = i / (Hq * 8);
      const int u = (int)(i - t * (Hq * 8)), h = u >> 3, v = (u & 7) * 8;
      const float4* src = reinterpret_cast<const float4*>(dq_acc + (t * Hq + h) * HD + v);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float4 x = src[j], y = src[16 + j];
        a[4 * j] = x.x; a[4 * j + 1] = x.y; a[4 * j + 2] = x.z; a[4 * j + 3] = x.w;
        z[4 * j] = y.x; z[4 * j + 1] = y.y; z[4 * j + 2] = y.z; z[4 * j + 3] = y.w;
      }
      store_gradient(dq + t * dq_stride + h * HD + v, a, z, rope_at(rope, (int)(t % S), v), scale);
    } else {  // a warp: eight keys x four groups of dims (whole lines read, 64 contiguous bytes per key written)
      const long long k = i - n_dq, block = k >> 10;
      const int v = ((int)k & 3) + ((int)(k >> 5) & 1) * 4, row = ((int)(k >> 2) & 7) + ((int)(k >> 6) & 15) * 8, is_v = (int)(block & 1);
      const long long bj = (block >> 1) / Hkv;
      const int hk = (int)((block >> 1) - bj * Hkv), s = (int)(bj % n_kt) * BKV + row;
      if (s >= S) continue;
      const float4* src = dkv_parts + block * PART_TILE + 2 * v * BKV + row;
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] = z[j] = 0.f;
      for (int p0 = 0; p0 < parts; p0 += 4, src += 4 * blocks * PART_TILE) {  // four parts in flight
        float4 x[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            x[p][j] = p0 + p < parts ? __ldcg(src + p * blocks * PART_TILE + ((j & 1) + (j >> 1) * 16) * BKV) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            a[4 * j] += x[p][j].x; a[4 * j + 1] += x[p][j].y; a[4 * j + 2] += x[p][j].z; a[4 * j + 3] += x[p][j].w;
            z[4 * j] += x[p][2 + j].x; z[4 * j + 1] += x[p][2 + j].y; z[4 * j + 2] += x[p][2 + j].z; z[4 * j + 3] += x[p][2 + j].w;
          }
      }
      __nv_bfloat16* dst = (is_v ? dv : dk) + ((bj / n_kt) * S + s) * dkv_stride + hk * HD + v * 8;
      store_gradient(dst, a, z, is_v ? nullptr : rope_at(rope, s, v * 8), is_v ? 1.f : scale);
    }
  }
}

// CTAs per key tile of a KV head.  With grouped-query attention a KV head's key tiles are few and their walks long (every
// query head of the group): the walk is cut by query heads where that is estimated to end sooner.  The main kernel takes its longest
// walk or its share of all steps, 1.5 us a step and 8 us a CTA (start, end, first loads); the parts' sums (131 KB a CTA) are read at
// 3.7 TB/s.  Measured, the whole backward pass, us, in 1 / 2 / 4 / 8 parts (* the choice):
//   1 x 333 tokens, 64 / 8 heads 88 / 56 / 42 / 42*;  1 x 777, 64 / 8 166 / 103 / 72* / 92;  1 x 2048, 64 / 8 396 / 253* / 290 / 331;
//   1 x 8192, 64 / 8 3422* / 3335 / 3455 / 3457;  8 x 300, 32 / 8 85* / 97 / 121;  4 x 1024, 32 / 8 162* / 204 / 255;
//   1 x 4096, 32 / 8 455 / 479* / 542;  1 x 4096, 28 / 4 653 whole, 432* in seven.
// (Cut until there were three CTAs per SM, 8 x 300 took 113, 4 x 1024 204 and 1 x 777 92 us.)
int head_parts_for(int B, int S, int Hq, int Hkv) {
  const int group = Hq / Hkv, n_kt = (S + BKV - 1) / BKV, n_qt = (S + BQ - 1) / BQ;
  const float sms = (float)yf_num_sms(), walks = (float)n_kt * (float)Hkv * (float)B;
  // steps of all walks, under the causal mask (key tile j starts at query tile 2 j)
  const float longest = (float)n_qt * (float)group;
  const float steps = (float)n_kt * (float)(n_qt - n_kt + 1) * (float)Hq * (float)B;
  int best = 1;
  float best_us = 0.f;
  for (int parts = 1; parts <= group; ++parts) {
    if (group % parts) continue;
    const float walk = longest / (float)parts * 1.5f + 8.f, share = (steps * 1.5f + walks * (float)parts * 8.f) / sms;
    const float us = (walk > share ? walk : share) + (parts > 1 ? walks * (float)parts * (131072.f / 3.7e6f) : 0.f);
    if (parts == 1 || us < best_us) {
      best = parts;
      best_us = us;
    }
  }
  return best;
}

}  // namespace

// The three launches of one backward pass (delta pre-pass, main kernel, dQ conversion), shared by both entry points.
// Allocates nothing: the tensor maps come by reference from the caller, the scratch by pointer.
static int attn_bwd_launch(int head_parts, float* dkv_parts, const float* rope, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& md,
                           const CUtensorMap& mdq, const void* out,
                           const void* dout, const float* lse, float* delta, float* dq_accum, void* dq, void* dk, void* dv, int B,
                           int S, int Hq, int Hkv, long long o_stride, long long do_stride, long long dq_stride,
                           long long dkv_stride, float scale, int causal, cudaStream_t st) {
  const auto kernel = dkv_parts != nullptr ? attn_bwd_kernel<true> : attn_bwd_kernel<false>;
  static bool optin[2][64] = {};  // the shared-memory opt-in is a per-device attribute
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  bool& done = optin[dkv_parts != nullptr ? 1 : 0][dev];
  if (!done) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, BWD_SMEM);
    if (e != cudaSuccess) return -(int)e;
    done = true;
  }
  if (int rc = yf_tu_bind_status()) return rc;
  const long long T = (long long)B * S;
  {
    // delta pre-pass; it also clears the dQ accumulator, which must start at zero on every call
    const long long groups = T * Hq;
    long long blocks = (groups * 16 + 255) / 256;
    const long long cap = (long long)yf_num_sms() * 8;
    if (blocks > cap) blocks = cap;
    attn_delta_kernel<<<(int)blocks, 256, 0, st>>>(reinterpret_cast<const __nv_bfloat16*>(out),
                                                  reinterpret_cast<const __nv_bfloat16*>(dout), delta, dq_accum, B, S, Hq,
                                                  o_stride, do_stride);
  }
  BwdArgs a;
  a.lse = lse;
  a.delta = delta;
  a.dkv_parts = reinterpret_cast<float4*>(dkv_parts);
  a.rope = rope;
  a.head_parts = head_parts;
  a.dk = reinterpret_cast<__nv_bfloat16*>(dk);
  a.dv = reinterpret_cast<__nv_bfloat16*>(dv);
  a.dkv_stride = dkv_stride;
  a.S = S; a.B = B; a.Hq = Hq; a.Hkv = Hkv;
  a.scale = scale;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.causal = causal ? 1 : 0;
  const int n_kt = (S + BKV - 1) / BKV;
  a.head_group = head_group_size(n_kt, B * Hkv * head_parts, T * Hq * HD * 4, yf_num_sms());  // the dQ accumulator
  const long long ctas = (long long)n_kt * B * Hkv * head_parts;
  if (ctas > 0x7fffffffll) return -1;
  const int grid = (int)ctas;
  kernel<<<grid, BWD_THREADS, BWD_SMEM, st>>>(mq, mk, mv, md, mdq, a);
  {
    const long long items = T * Hq * 8 + (dkv_parts ? (long long)B * n_kt * Hkv * 2 * BKV * 8 : 0);
    long long blocks = (items + 255) / 256;
    const long long cap = (long long)yf_num_sms() * 8;
    if (blocks > cap) blocks = cap;
    attn_convert_kernel<<<(int)blocks, 256, 0, st>>>(dq_accum, a.dkv_parts, head_parts, rope, reinterpret_cast<__nv_bfloat16*>(dq), a.dk, a.dv, B, S, Hq, Hkv,
                                                     dq_stride, dkv_stride, scale);
  }
  return -(int)cudaGetLastError();
}

// Backward of yf_attn_fwd.  q/k/v/out/dout as in the forward (dout rows do_stride apart, out rows
// o_stride apart); lse from the forward.  Scratch supplied by the caller: delta [B,Hq,S] fp32 and
// dq_accum [B*S, Hq*128] fp32 (zeroed here).  Results: dq (rows dq_stride apart), dk/dv (rows
// dkv_stride apart), all bf16; they may be column blocks of one fused d(QKV) buffer.
// The general form: `dkv_parts` (scratch of head_parts * 2 * B * S rounded up to 128 * Hkv * 128 floats, whose contents do not matter; dkv_floats says
// how many there are) lets `head_parts` CTAs (a divisor of Hq / Hkv) share a key tile of a KV head; yf_attn_bwd_head_parts says how many a
// problem wants.  head_parts == 1 takes none.  dK and dV do not vary from run to run (dQ's atomic sums may).  `rope` (may be
// null; [S, 64, 2] fp32 cos, sin, 16-byte aligned): q and k are rotated, dq and dk are wanted with respect to what was rotated.
extern "C" int yf_attn_bwd_head_parts(int B, int S, int Hq, int Hkv) {
  if (B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || (Hq % Hkv)) return -1;
  return head_parts_for(B, S, Hq, Hkv);
}
extern "C" int yf_attn_bwd_parts(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                                 float* delta, float* dq_accum, float* dkv_parts, long long dkv_floats, int head_parts, const float* rope, void* dq, void* dk, void* dv, int B,
                                 int S, int Hq, int Hkv, long long q_stride, long long kv_stride, long long o_stride,
                                 long long do_stride, long long dq_stride, long long dkv_stride, float scale, int causal, void* stream) {
  if (B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || (Hq % Hkv)) return -1;
  if (head_parts < 1 || (Hq / Hkv) % head_parts || (head_parts > 1) != (dkv_parts != nullptr)) return -1;
  if (dkv_parts != nullptr && dkv_floats < 4 * part_tile(head_parts, B, 0, (S + BKV - 1) / BKV, 0, Hkv, 0, 0)) return -1;
  if ((q_stride % 8) || (kv_stride % 8) || (o_stride % 8) || (do_stride % 8) || (dq_stride % 8) || (dkv_stride % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dq) |
       reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv) | reinterpret_cast<uintptr_t>(dq_accum) |
       reinterpret_cast<uintptr_t>(dkv_parts) | reinterpret_cast<uintptr_t>(rope)) & 15)
    return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  const CUtensorMap* mq = yf_tensor_map_3d(q, (uint64_t)Hq * HD, S, B, q_stride, (uint64_t)S * q_stride, 64, BQ, 1, 2, 1);
  const CUtensorMap* mk = yf_tensor_map_3d(k, (uint64_t)Hkv * HD, S, B, kv_stride, (uint64_t)S * kv_stride, 64, BKV, 1, 2, 1);
  const CUtensorMap* mv = yf_tensor_map_3d(v, (uint64_t)Hkv * HD, S, B, kv_stride, (uint64_t)S * kv_stride, 64, BKV, 1, 2, 1);
  const CUtensorMap* md = yf_tensor_map_3d(dout, (uint64_t)Hq * HD, S, B, do_stride, (uint64_t)S * do_stride, 64, BQ, 1, 2, 1);
  const CUtensorMap* mdq = yf_tensor_map_3d(dq_accum, (uint64_t)Hq * HD, S, B, (uint64_t)Hq * HD, (uint64_t)S * Hq * HD, 32, BQ, 1, 4, 0);
  if (!mq || !mk || !mv || !md || !mdq) return -2;
  return attn_bwd_launch(head_parts, dkv_parts, rope, *mq, *mk, *mv, *md, *mdq, out, dout, lse, delta, dq_accum, dq, dk, dv, B, S, Hq, Hkv,
                         o_stride, do_stride, dq_stride, dkv_stride, scale, causal, st);
}
extern "C" int yf_attn_bwd(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                           float* delta, float* dq_accum, void* dq, void* dk, void* dv, int B, int S, int Hq, int Hkv,
                           long long q_stride, long long kv_stride, long long o_stride, long long do_stride,
                           long long dq_stride, long long dkv_stride, float scale, int causal, void* stream) {
  return yf_attn_bwd_parts(q, k, v, out, dout, lse, delta, dq_accum, nullptr, 0, 1, nullptr, dq, dk, dv, B, S, Hq, Hkv, q_stride, kv_stride, o_stride,
                           do_stride, dq_stride, dkv_stride, scale, causal, stream);
}

// ------------------------------------------------------------------------------------------------
// yf_attn_bwd_noalloc: the same backward for callers that cannot allocate device memory.
//
// yf_attn_bwd needs two scratch arrays from its caller (delta and the fp32 dQ accumulator).  Some users of
// this library have no way to provide them: a C or C++ host that binds the exported symbols without a
// tensor framework, or a job that hands all of the GPU's memory to its own pool at start-up, where a later
// cudaMalloc fails and a borrowed pool block is not available to a third-party call.  For them the scratch
// lives in the fixed device array below, which every GPU that loads this library holds until the process
// exits (about 16.1 MiB).  Nothing here calls cudaMalloc, cudaFree, a framework allocator or the tensor-map
// cache (the descriptors are encoded into stack storage).
//
// Limits and rules:
//  * B * S * Hq must not exceed YF_ATTN_NOALLOC_MAX_ROWS (32768 query rows x heads, e.g. one 2048-token
//    sequence with 16 heads); larger problems are refused with -3 and a message on stderr.
//  * The first call on each device looks up the array's device address (cudaGetSymbolAddress, with that
//    device current).  Make that first call outside of any stream capture.
//  * All calls on a device share the one array and it keeps the previous call's contents; the part that must
//    start at zero (the dQ accumulator) is cleared by every call.  Two calls whose kernels overlap on the GPU
//    (different streams) race on it: keep calls on one device ordered.
//
// In host code the array's name is only a stand-in for the symbol, not a device address, so the host never
// passes it to a kernel: it passes the pointer that cudaGetSymbolAddress returned.
constexpr long long YF_ATTN_NOALLOC_MAX_ROWS = 32768;
constexpr long long NOALLOC_DELTA_FLOATS = YF_ATTN_NOALLOC_MAX_ROWS;                 // delta [B, Hq, S]
constexpr long long NOALLOC_DQ_FLOATS = YF_ATTN_NOALLOC_MAX_ROWS * 128;              // dQ accumulator [B*S, Hq*128]
static __device__ __align__(256) float g_attn_noalloc_scratch[NOALLOC_DELTA_FLOATS + NOALLOC_DQ_FLOATS];

static float* attn_noalloc_scratch_for_current_device(int* err) {
  static float* ptrs[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    *err = e != cudaSuccess ? -(int)e : -1;
    return nullptr;
  }
  if (ptrs[dev] == nullptr) {
    float* p = nullptr;
    e = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_attn_noalloc_scratch);
    if (e != cudaSuccess || p == nullptr) {
      *err = e != cudaSuccess ? -(int)e : -1;
      return nullptr;
    }
    ptrs[dev] = p;
  }
  *err = 0;
  return ptrs[dev];
}

extern "C" int yf_attn_bwd_noalloc(const void* q, const void* k, const void* v, const void* out, const void* dout, const float* lse,
                                   void* dq, void* dk, void* dv, int B, int S, int Hq, int Hkv, long long q_stride,
                                   long long kv_stride, long long o_stride, long long do_stride, long long dq_stride,
                                   long long dkv_stride, float scale, int causal, void* stream) {
  if (B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || (Hq % Hkv)) return -1;
  if ((q_stride % 8) || (kv_stride % 8) || (o_stride % 8) || (do_stride % 8) || (dq_stride % 8) || (dkv_stride % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(dout) | reinterpret_cast<uintptr_t>(dq) |
       reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 15)
    return -1;
  const long long rows = (long long)B * S * Hq;
  if (rows > YF_ATTN_NOALLOC_MAX_ROWS) {
    fprintf(stderr,
            "[yafsdp_b200] yf_attn_bwd_noalloc: B*S*Hq = %lld exceeds the built-in scratch for %lld rows; "
            "use yf_attn_bwd with caller-provided scratch\n",
            rows, YF_ATTN_NOALLOC_MAX_ROWS);
    return -3;
  }
  int err = 0;
  float* scratch = attn_noalloc_scratch_for_current_device(&err);
  if (scratch == nullptr) return err;
  float* delta = scratch;
  float* dq_accum = scratch + NOALLOC_DELTA_FLOATS;  // 131072 bytes in: still 256-byte aligned
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  CUtensorMap mq, mk, mv, md, mdq;  // encoded in place: the cached variants would allocate a cache entry
  if (yf_tensor_map_3d_encode(&mq, q, (uint64_t)Hq * HD, S, B, q_stride, (uint64_t)S * q_stride, 64, BQ, 1, 2, 1) != 0 ||
      yf_tensor_map_3d_encode(&mk, k, (uint64_t)Hkv * HD, S, B, kv_stride, (uint64_t)S * kv_stride, 64, BKV, 1, 2, 1) != 0 ||
      yf_tensor_map_3d_encode(&mv, v, (uint64_t)Hkv * HD, S, B, kv_stride, (uint64_t)S * kv_stride, 64, BKV, 1, 2, 1) != 0 ||
      yf_tensor_map_3d_encode(&md, dout, (uint64_t)Hq * HD, S, B, do_stride, (uint64_t)S * do_stride, 64, BQ, 1, 2, 1) != 0 ||
      yf_tensor_map_3d_encode(&mdq, dq_accum, (uint64_t)Hq * HD, S, B, (uint64_t)Hq * HD, (uint64_t)S * Hq * HD, 32, BQ, 1, 4, 0) != 0)
    return -2;
  return attn_bwd_launch(1, nullptr, nullptr, mq, mk, mv, md, mdq, out, dout, lse, delta, dq_accum, dq, dk, dv, B, S, Hq, Hkv, o_stride, do_stride, dq_stride,
                         dkv_stride, scale, causal, st);
}
