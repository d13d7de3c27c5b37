// Causal flash-attention forward for head_dim 128 on sm_100a (MHA and GQA).
//
// One CTA per (256 query rows, query head, sequence), as two tiles of 128 rows that take turns on the tensor cores (one
// tile where the whole problem then still fits the GPU at once).  Roles:
//   warp 0      TMA producer: Q once, then K/V tiles of 128 keys through a 2-stage ring
//   warp 1      MMA issuer:   S_i = Q_i K^T and O_i += P_i V for the tiles i = 0, 1
//   warps 2-5   softmax of tile 0, warps 6-9 of tile 1: one thread per query row (TMEM lane == row)
// While one tile's softmax runs, the tensor cores work for the other one.  TMEM (512 columns): S_0, S_1, O_0, O_1, 128
// columns of fp32 each; P_i (bf16, 64 columns) takes the place of S_i, whose row its thread has read into registers, and is
// the MMA's A operand from there, so the probabilities never go through shared memory.  A row belongs to one thread: the
// softmax threads exchange nothing but one bit per block, at a barrier of the tile's four warps (below).
// The output accumulates in TMEM over all key blocks (O += P V).  The exponent's reference maximum is only moved when
// some row of a tile has grown by more than 2^8 since it was set (then its warps rescale their rows of O in TMEM and their
// sums); otherwise P is taken relative to the older maximum (values up to 2^8, harmless in bf16 / fp32), and the final
// division by the row sum makes the result exact again.
// Bound: per 128 x 128 block the two MMAs take 1024 cycles and the 16 384 exponentials at 16 per cycle as long, on
// different pipes.
// Inputs are read in place from the fused QKV projection output ([tokens, (Hq+2Hkv)*128], row pitch
// given), so no head transposes are materialised.  Writes O (bf16) and the log-sum-exp per row (fp32).
#include "common.cuh"
#include "yafsdp_b200.h"

YF_TU_STATUS()

namespace {

constexpr int HD = 128;        // head dim
constexpr int BQ = 128;        // query rows per tile
constexpr int BKV = 128;       // keys per tile
constexpr int ATOM = 16384;    // bytes of one [128 rows x 64 bf16] swizzled block
constexpr int TILE = 2 * ATOM; // one 128x128 bf16 tile
constexpr int FWD_THREADS = 320;  // producer warp, MMA warp, eight softmax warps
constexpr int FWD_SMEM = 1024 + 2 * TILE /*Q*/ + 2 * 2 * TILE /*K,V x2 stages*/ + 256;

struct FwdArgs {
  __nv_bfloat16* out;
  float* lse;
  long long out_stride;  // elements between token rows of out
  int S, B, Hq, Hkv;
  float scale_log2;      // softmax scale * log2(e)
  float scale;
  int causal;
  int tiles;             // query tiles per CTA: two, or one where even so every CTA finds an SM of its own
};

__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tma_q, const __grid_constant__ CUtensorMap tma_k,
                const __grid_constant__ CUtensorMap tma_v, FwdArgs args) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sQ = smem;                   // tile i at + i * TILE
  uint8_t* sKV = sQ + 2 * TILE;         // stage s: K at sKV + s*2*TILE, V at + TILE
  uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + 4 * TILE);
  uint64_t* q_full = bars;              // [2] per tile
  uint64_t* k_full = bars + 2;          // [2] per stage
  uint64_t* v_full = bars + 4;          // [2]
  uint64_t* k_empty = bars + 6;         // [2]
  uint64_t* v_empty = bars + 8;         // [2]
  uint64_t* s_full = bars + 10;         // [2] per tile
  uint64_t* p_ready = bars + 12;        // [2] per tile
  uint64_t* o_full = bars + 14;         // [2] per tile
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_slot + 1);  // [2] per tile: 1 + the block at which one of its warps has given up

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // the query position is the slowest index: under the causal mask the long rows of all heads start first
  const int qt = args.causal ? (int)(gridDim.z - 1 - blockIdx.z) : (int)blockIdx.z;
  const int h = blockIdx.x;
  const int b = blockIdx.y;
  const int hkv = h / (args.Hq / args.Hkv);
  const int q0 = qt * args.tiles * BQ;
  const int n_kv_total = (args.S + BKV - 1) / BKV;
  // key blocks of the two tiles (the second one has none when the sequence ends in the first, or a CTA has one tile)
  const int n_kv0 = args.causal ? min(q0 / BKV + 1, n_kv_total) : n_kv_total;
  const int n_kv1 = args.tiles < 2 || q0 + BQ >= args.S ? 0 : (args.causal ? min(q0 / BKV + 2, n_kv_total) : n_kv_total);
  const int n_kv = max(n_kv0, n_kv1);

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tma_q);
    tma_prefetch_desc(&tma_k);
    tma_prefetch_desc(&tma_v);
    for (int s = 0; s < 2; ++s) {
      mbar_init(&q_full[s], 1);
      mbar_init(&k_full[s], 1);
      mbar_init(&v_full[s], 1);
      mbar_init(&k_empty[s], 1);
      mbar_init(&v_empty[s], 1);
      mbar_init(&s_full[s], 1);
      mbar_init(&p_ready[s], 4);  // one arrival per softmax warp of the tile
      mbar_init(&o_full[s], 1);
      dead[s] = 0;
    }
    mbar_fence_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(&q_full[0], TILE);
      tma_load_3d(sQ, &tma_q, &q_full[0], h * HD, q0, b);
      tma_load_3d(sQ + ATOM, &tma_q, &q_full[0], h * HD + 64, q0, b);
      for (int j = 0; j < n_kv; ++j) {
        const int s = j & 1;
        uint8_t* sK = sKV + s * 2 * TILE;
        uint8_t* sV = sK + TILE;
        if (!mbar_wait(&k_empty[s], ((j >> 1) & 1) ^ 1, 100)) break;
        mbar_expect_tx(&k_full[s], TILE);
        tma_load_3d(sK, &tma_k, &k_full[s], hkv * HD, j * BKV, b);
        tma_load_3d(sK + ATOM, &tma_k, &k_full[s], hkv * HD + 64, j * BKV, b);
        if (j == 0 && n_kv1 > 0) {
          mbar_expect_tx(&q_full[1], TILE);
          tma_load_3d(sQ + TILE, &tma_q, &q_full[1], h * HD, q0 + BQ, b);
          tma_load_3d(sQ + TILE + ATOM, &tma_q, &q_full[1], h * HD + 64, q0 + BQ, b);
        }
        if (!mbar_wait(&v_empty[s], ((j >> 1) & 1) ^ 1, 101)) break;
        mbar_expect_tx(&v_full[s], TILE);
        tma_load_3d(sV, &tma_v, &v_full[s], hkv * HD, j * BKV, b);
        tma_load_3d(sV + ATOM, &tma_v, &v_full[s], hkv * HD + 64, j * BKV, b);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc_s = umma_idesc_bf16(BQ, BKV, 0, 0);   // Q, K both K-major (K = head dim)
      const uint32_t idesc_o = umma_idesc_bf16(BQ, HD, 0, 1);    // P from TMEM (K = keys), V MN-major
      const uint64_t dQ = umma_smem_desc_sw128(smem_u32(sQ), 0, 1024);
      const uint64_t dK = umma_smem_desc_sw128(smem_u32(sKV), 0, 1024);
      const uint64_t dV = umma_smem_desc_sw128(smem_u32(sKV) + TILE, ATOM, 1024);
      // descriptor addresses advance in units of 16 bytes
      auto issue_s = [&](int i, int j) {
        const uint64_t q = dQ + i * (TILE >> 4), k = dK + (j & 1) * (2 * TILE >> 4);
#pragma unroll
        for (int e = 0; e < HD / 16; ++e) {
          const uint32_t off = ((e >> 2) * ATOM + (e & 3) * 32) >> 4;
          tc_mma_bf16(tmem_base + i * 128, q + off, k + off, idesc_s, e != 0);
        }
        tc_commit(&s_full[i]);
      };
      auto issue_o = [&](int i, int j) {
        const uint64_t v = dV + (j & 1) * (2 * TILE >> 4);
#pragma unroll
        for (int e = 0; e < BKV / 16; ++e)  // 16 keys: 8 TMEM columns of P, 16 rows of V
          tc_mma_bf16_ts(tmem_base + 256 + i * 128, tmem_base + i * 128 + e * 8, v + e * (2048 >> 4), idesc_o, (j | e) != 0);
        tc_commit(&o_full[i]);
      };
      bool alive = mbar_wait(&k_full[0], 0, 110) && mbar_wait(&q_full[0], 0, 111);
      if (alive) {
        tc_fence_after();
        issue_s(0, 0);
        if (n_kv1 > 0 && (alive = mbar_wait(&q_full[1], 0, 112))) {
          tc_fence_after();
          issue_s(1, 0);
        }
        tc_commit(&k_empty[0]);
      }
      for (int j = 0; j < n_kv && alive; ++j) {
        const int s = j & 1;
        if (j + 1 < n_kv && !mbar_wait(&k_full[s ^ 1], ((j + 1) >> 1) & 1, 113)) break;
        if (!mbar_wait(&v_full[s], (j >> 1) & 1, 114)) break;
        // P_i(j) V, then S_i(j+1) into the columns that P_i(j) held: the order of MMAs with different accumulators is not
        // promised, so the product is waited for (about 200 cycles; the other tile's softmax is running meanwhile)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int n = i == 0 ? n_kv0 : n_kv1;
          if (j >= n) continue;
          if (!mbar_wait(&p_ready[i], j & 1, 115 + i)) { alive = false; break; }
          tc_fence_after();
          issue_o(i, j);
          if (j + 1 < n) {
            if (!mbar_wait(&o_full[i], j & 1, 117 + i)) { alive = false; break; }
            tc_fence_after();
            issue_s(i, j + 1);
          }
        }
        if (j + 1 < n_kv) tc_commit(&k_empty[s ^ 1]);
        tc_commit(&v_empty[s]);
      }
    }
  } else {
    const int i = (warp - 2) >> 2;           // tile
    const int n = i == 0 ? n_kv0 : n_kv1;
    const int q = warp & 3;                  // a warp may only touch TMEM lanes [32*(warp%4), +32)
    const int qrow = q0 + i * BQ + q * 32 + lane;
    const uint32_t lane_off = (uint32_t)(q * 32) << 16;
    const uint32_t tS = tmem_base + lane_off + i * 128, tO = tmem_base + lane_off + 256 + i * 128;
    float m_run = -INFINITY;                 // reference maximum of the exponent
    float l_run[2] = {0.f, 0.f};             // row sums of the even and the odd 64 keys of all blocks, each in the order of the keys
    const float sl2 = args.scale_log2;
    constexpr float RESCALE_LOG2 = 8.f;      // move the reference maximum when a row's maximum exceeds it by 2^8
    // keys allowed for this row: col <= limit
    const int limit = args.causal ? min(qrow, args.S - 1) : (args.S - 1);
    bool alive = true;
    for (int j = 0; j < n; ++j) {
      // a bounded wait that runs out ends the work of the tile's four warps: they meet at the barrier below, so the one that gives up
      // says so there (the lanes of a warp decide together: TMEM accesses are warp-wide)
      alive = alive && __all_sync(0xffffffffu, mbar_wait(&s_full[i], j & 1, 120 + i));
      const int kv0 = j * BKV;
      uint32_t sc[4][32];
      if (alive) {
        tc_fence_after();
#pragma unroll
        for (int c = 0; c < 4; ++c) tmem_ld32(tS + c * 32, sc[c]);
        tmem_ld_wait();
      } else {
        dead[i] = j + 1;
      }
      if (kv0 + BKV - 1 > limit) {  // only the blocks on the diagonal and the last one have masked keys
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int t = 0; t < 32; ++t)
            if (kv0 + c * 32 + t > limit) sc[c][t] = 0xff800000u;  // -inf
      }
      float mx4[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        mx4[c] = __uint_as_float(sc[c][0]);
#pragma unroll
        for (int t = 1; t < 32; ++t) mx4[c] = fmaxf(mx4[c], __uint_as_float(sc[c][t]));
      }
      const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
      const bool grew = !alive || j == 0 || (mx != -INFINITY && (m_run == -INFINITY || (mx - m_run) * sl2 > RESCALE_LOG2));
      // The four warps of a tile move their rows' maxima together: a row's bits then depend on its tile alone and repeat those of
      // kernels that deal the rows to warps in another way.  The barrier costs 4 % at 2048 tokens x 32 heads (49 -> 51 us) and 8 % at
      // 8192 x 32/8 (570 -> 615 us), less than 0.2 % of a layer's forward and backward.
      if (i == 0 ? named_bar_or(1, 128, grew) : named_bar_or(2, 128, grew)) {
        if (dead[i] == j + 1) { alive = false; break; }  // not a later block's: who gives up there waits for this warp there
        const float m_new = fmaxf(m_run, mx);
        if (j > 0) {
          // O holds sums relative to the old maximum: wait for the last P V to land, then scale this warp's rows
          alive = __all_sync(0xffffffffu, mbar_wait(&o_full[i], (j - 1) & 1, 122 + i));
          if (!alive) continue;  // to the next barrier, where the others learn of it
          tc_fence_after();
          const float alpha = (m_run == -INFINITY) ? 0.f : fast_exp2((m_run - m_new) * sl2);
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t r[32];
            tmem_ld32(tO + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int t = 0; t < 32; ++t) r[t] = __float_as_uint(__uint_as_float(r[t]) * alpha);
            tmem_st32(tO + c * 32, r);
          }
          l_run[0] *= alpha;
          l_run[1] *= alpha;
        }
        m_run = m_new;
      }
      const float neg_ms = (m_run == -INFINITY) ? 0.f : -m_run * sl2;
#pragma unroll
      for (int c = 0; c < 2; ++c) {  // 64 keys: 32 TMEM columns of packed bf16 pairs
        uint32_t packed[32];
        float sum = 0.f;
#pragma unroll
        for (int t = 0; t < 32; ++t) {
          const float p0 = fast_exp2(fmaf(__uint_as_float(sc[2 * c + (t >> 4)][(2 * t) & 31]), sl2, neg_ms));
          const float p1 = fast_exp2(fmaf(__uint_as_float(sc[2 * c + (t >> 4)][(2 * t + 1) & 31]), sl2, neg_ms));
          sum += p0 + p1;  // one chain: an addition takes less than the two exponentials next to it
          packed[t] = pack_bf16x2(p0, p1);
        }
        tmem_st32(tS + c * 32, packed);
        l_run[c] += sum;
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[i]);
    }
    // the output of the last block
    if (n > 0 && alive && __all_sync(0xffffffffu, mbar_wait(&o_full[i], (n - 1) & 1, 124 + i))) {
      tc_fence_after();
      const float l = l_run[0] + l_run[1];
      const float inv = (l > 0.f) ? 1.f / l : 0.f;
      __nv_bfloat16* dst = args.out + ((long long)b * args.S + qrow) * args.out_stride + h * HD;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld32(tO + c * 32, r);
        tmem_ld_wait();
        if (qrow < args.S) {
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(r[8 * v + 0]) * inv, __uint_as_float(r[8 * v + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(r[8 * v + 2]) * inv, __uint_as_float(r[8 * v + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(r[8 * v + 4]) * inv, __uint_as_float(r[8 * v + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(r[8 * v + 6]) * inv, __uint_as_float(r[8 * v + 7]) * inv);
            reinterpret_cast<uint4*>(dst + c * 32)[v] = w;
          }
        }
      }
      if (qrow < args.S)
        args.lse[((long long)b * args.Hq + h) * args.S + qrow] = (l > 0.f) ? (m_run * args.scale + logf(l)) : -INFINITY;
    }
    tc_fence_before();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// q, k, v: bf16 pointers to the first head's first column; token rows are q_stride / kv_stride elements
// apart (the three may alias one fused projection output).  Tokens are ordered [batch, seq].
// out: [B*S, out_stride] bf16 (head h at columns h*128), lse: [B, Hq, S] fp32.
extern "C" int yf_attn_fwd(const void* q, const void* k, const void* v, void* out, float* lse, int B, int S, int Hq,
                           int Hkv, long long q_stride, long long kv_stride, long long out_stride, float scale, int causal,
                           void* stream) {
  if (B <= 0 || S <= 0 || Hq <= 0 || Hkv <= 0 || (Hq % Hkv) || (q_stride % 8) || (kv_stride % 8) || (out_stride % 8)) return -1;
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) |
       reinterpret_cast<uintptr_t>(out)) & 15)
    return -1;
  const CUtensorMap* mq = yf_tensor_map_3d(q, (uint64_t)Hq * HD, S, B, q_stride, (uint64_t)S * q_stride, 64, BQ, 1, 2, 1);
  const CUtensorMap* mk = yf_tensor_map_3d(k, (uint64_t)Hkv * HD, S, B, kv_stride, (uint64_t)S * kv_stride, 64, BKV, 1, 2, 1);
  const CUtensorMap* mv = yf_tensor_map_3d(v, (uint64_t)Hkv * HD, S, B, kv_stride, (uint64_t)S * kv_stride, 64, BKV, 1, 2, 1);
  if (!mq || !mk || !mv) return -2;
  static bool optin[64] = {};  // the shared-memory opt-in is a per-device attribute
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!optin[dev]) {
    cudaError_t e = cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
    if (e != cudaSuccess) return -(int)e;
    optin[dev] = true;
  }
  if (int rc = yf_tu_bind_status()) return rc;
  FwdArgs a;
  a.out = reinterpret_cast<__nv_bfloat16*>(out);
  a.lse = lse;
  a.out_stride = out_stride;
  a.S = S; a.B = B; a.Hq = Hq; a.Hkv = Hkv;
  a.scale = scale;
  a.scale_log2 = scale * 1.4426950408889634f;
  a.causal = causal ? 1 : 0;
  a.tiles = (long long)((S + BQ - 1) / BQ) * Hq * B <= yf_num_sms() ? 1 : 2;
  dim3 grid(Hq, B, (S + a.tiles * BQ - 1) / (a.tiles * BQ));
  attn_fwd_kernel<<<grid, FWD_THREADS, FWD_SMEM, reinterpret_cast<cudaStream_t>(stream)>>>(*mq, *mk, *mv, a);
  return -(int)cudaGetLastError();
}
