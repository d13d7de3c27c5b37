// bf16 GEMM family for sm_100a: C[M,N] = alpha * A[M,K] * B[N,K]^T (+ C), fp32 accumulation in TMEM.
//
// Persistent, warp-specialised kernel, one CTA per SM:
//   warp 0     TMA producer  (cp.async.bulk.tensor, 128-byte swizzle, no multicast); plain modes: warps 0 and 6 in turn
//   warp 1     MMA issuer    (tcgen05.mma, 128 rows per CTA, cta_group::1 or one instruction for a pair of CTAs, K=16)
//   warps 2-5  epilogue      (tcgen05.ld 32x32b, convert, store; overlaps the next tile's main loop
//                             through two TMEM accumulators)
// Either operand may be K-major (rows of K contiguous) or MN-major (the M/N index contiguous), so
// the three GEMMs of a linear layer (Y = X W^T, dX = dY W, dW = dY^T X) run without a transpose.
// The fp32 output mode with accumulate writes weight gradients straight into a flat fp32 gradient
// buffer (the cast and the micro-batch accumulation of a sharded-data-parallel step).
#include <limits.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <numeric>
#include <utility>

#include "common.cuh"
#include "yafsdp_b200.h"

YF_TU_STATUS()

namespace {

constexpr int BLOCK_M = 128;
constexpr int BLOCK_K = 64;   // 64 bf16 = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int GEMM_THREADS = 192;
constexpr int WIDE_THREADS = 224;  // one more warp: plain mode's second TMA producer, gather mode's communication role

// MODE_PLAIN: C is stored locally through TMA; MODE_SPLIT: so too, and the last wave's tiles are split along K (an
// instantiation of its own: the exchange's code alone costs the plain kernel 0.3 us per tile).
// MODE_SCATTER: GEMM -> reduce-scatter, the fp32 rows of C are pushed to the ranks that own them.  MODE_GATHER: all-gather ->
// GEMM, the kernel also gathers the layer that B is part of (see FusedArgs).
// MODE_SWIGLU: the gate and up projections of an MLP with their activation (see GemmArgs).
// MODE_SWAP: C is stored transposed: A is the weight, B the tokens, whose tile is any multiple of 16 wide (see GemmArgs::bn).
constexpr int MODE_PLAIN = 0, MODE_SCATTER = 1, MODE_GATHER = 2, MODE_SPLIT = 3, MODE_SWIGLU = 4, MODE_SWAP = 5;
__host__ __device__ constexpr bool is_plain(int mode) { return mode != MODE_SCATTER && mode != MODE_GATHER; }
constexpr int SCATTER_COLS = 64;                         // columns per pushed row piece: 256 bytes of fp32
constexpr int SCATTER_PITCH = SCATTER_COLS * 4 + 16;     // row pitch of the staging block (16 B of padding: no bank conflicts)

template <int BLOCK_N, int CG, int MODE = MODE_PLAIN>
struct GemmCfg {
  static constexpr int B_ROWS = BLOCK_N / CG;  // rows of B (N extent) in one CTA's shared memory
  static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2;
  static constexpr int B_BYTES = B_ROWS * BLOCK_K * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int RING_BYTES = (MODE == MODE_GATHER) ? 6 * 16384 : 0;  // the communication role's ring (COMM_SLOTS pieces)
  static constexpr int STAGES = (MODE == MODE_SCATTER) ? (STAGE_BYTES == 49152 ? 3 : 4)
                                : (MODE == MODE_GATHER) ? (STAGE_BYTES == 49152 ? 2 : 3)
                                                        : 196608 / STAGE_BYTES;  // 192 KB of operands in flight
  static constexpr int TMEM_COLS = 2 * BLOCK_N;  // two accumulators (a power of two)
  // plain: two [32 rows x 128 B] swizzled blocks per warp for TMA stores; scatter: two [128 rows x 256 B (+ padding)] linear blocks
  static constexpr int STAGING_BYTES = (MODE == MODE_SCATTER) ? 2 * BLOCK_M * SCATTER_PITCH : 2 * 16384 + RING_BYTES;
  static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + STAGING_BYTES + 256;
};

constexpr int MAX_SPLITS = 4;  // K ranges of one tile (split mode)

constexpr int MAX_RANKS = 16;
constexpr int MAX_GROUP = 4;  // problems of one grouped launch (the weight-gradient GEMMs of a decoder layer)

struct GemmArgs {
  void* C;
  int M, N, K;
  long long ldc;
  float alpha;
  const float* alpha_ptr;  // optional: one fp32 on the device that alpha is multiplied by
  int a_mn, b_mn, out_f32, accumulate;
  // optional bf16 residual [M, N] with row pitch ldr, added in fp32 before the bf16 output is rounded (bf16 output, plain
  // mode): a block's "x + proj(...)" costs no pass of its own over the activations
  const void* R;
  long long ldr;
  // MODE_SWIGLU: B is two matrices of N / 2 rows, gate (maps.b[0]) and up (maps.b[1]); a tile is 128 columns of each, and the
  // epilogue writes silu(gate) * up, of the values as rounded to bf16, through maps.a[1] and, with store_gu, gate and up into
  // the halves of C.
  int store_gu;
  // MODE_SWAP: M counts the output's columns (rows of the weight, operand A) and N its rows (tokens, operand B), so that the
  // padding of a ragged number of tokens shrinks from a multiple of 256 to one of 16 and the width of a tile can be chosen for
  // full waves.  bn: tokens per tile, half of them in each CTA of the pair.
  int bn;
  // B (MODE_SWAP: A) in several pieces of memory (plain modes): parts[i] is where piece i ends, in rows of [N, K] storage (then no
  // tile crosses a piece's end) or of [K, N] storage (no K block does).  n_parts <= 1: one piece.
  int n_parts;
  int parts[MAX_GROUP];
  // Split tiles (split mode).  The number of tiles modulo the number of units is what a last wave would leave most units
  // idle for: so many tiles, [0, split_tiles), are computed in `splits` K ranges each, the others whole.  Work items are
  // dealt round-robin: range 0 of every split tile, range 1 of every split tile, and so on - the units that run at the same
  // time read the same part of K (L2) - and then the whole tiles, whose main loops hide the exchange of the sums.  A
  // range's fp32 sums go to its slot of `slots` ([128 rows x BLOCK_N] per CTA); the CTA that arrives last at the tile's
  // counter adds the ranges in their order (the result does not depend on which one that is) and writes the output.
  // Nobody waits.  A counter is (nonce << 8 | arrivals): the nonce is new in every launch, so what the workspace held
  // before does not matter and nothing has to be cleared; the last one leaves a zero (replays of a captured launch).
  int split_tiles, splits;
  unsigned long long nonce;
  unsigned long long* counters;
  float* slots;
  // Grouped launch (scatter mode): n_prob problems that share K and the operand majors, in the order of their positions in
  // the flat layer gradient.  Tiles are numbered problem by problem, rows first (= in flat order); tile_prefix[p] = number
  // of tiles in front of problem p; own_start[o] = first tile whose rows begin in the shard of rank o.  The launch deals the
  // owners' tiles round-robin, starting with the rank after this one: step t works on tile t / world of owner
  // (rank + 1 + t % world) % world, so every rank pushes to all owners (and computes for itself) all the time and no
  // owner's NVLink ingress becomes a hot spot whatever the skew between the ranks.  n_prob == 0: one problem, M x N above.
  int n_prob;
  int Mp[MAX_GROUP], Np[MAX_GROUP];
  long long flat_off[MAX_GROUP];
  int tile_prefix[MAX_GROUP + 1];
  int own_start[MAX_RANKS + 1];
  int steps;   // world * (largest number of tiles of one owner)
};

// the factor of A * B^T, possibly with a device scalar in it
YF_DEVINL float alpha_of(const GemmArgs& args) { return args.alpha_ptr != nullptr ? args.alpha * __ldg(args.alpha_ptr) : args.alpha; }

// one piece of work of a unit: K blocks [kb0, kb1) of a tile; part < 0: all of them
struct WorkItem {
  int tile, kb0, kb1, part;
};
template <int MODE>
YF_DEVINL WorkItem work_item(const GemmArgs& args, int i, int num_k) {
  WorkItem w = {i, 0, num_k, -1};
  if constexpr (MODE == MODE_SPLIT) {
    if (i < args.split_tiles * args.splits) {
      w.part = i / args.split_tiles;
      w.tile = i - w.part * args.split_tiles;
      w.kb0 = (int)((long long)num_k * w.part / args.splits);
      w.kb1 = (int)((long long)num_k * (w.part + 1) / args.splits);
    } else {
      w.tile = i - args.split_tiles * (args.splits - 1);
    }
  }
  return w;
}

// operand tensor maps of up to MAX_GROUP problems (entry 0 alone for an ordinary launch)
struct GroupMaps {
  CUtensorMap a[MAX_GROUP], b[MAX_GROUP];
};

// Arguments of the two fused compute + collective modes (both off when zero-initialised).
//
// gather (all-gather -> GEMM, MODE_GATHER): every CTA of the GEMM carries one extra warp whose elected thread pulls its
// share of every rank's bf16 shard of the layer (bulk loads from peer memory over NVLink into a small ring in shared
// memory, bulk stores from there into the local layer buffer) and, for every piece that lies inside B, adds the piece's
// bytes to the counter of the B column block it belongs to.  The producer warps wait (bounded) until the counter of a tile's
// column block says that all of its rows have landed, then load B from the local buffer as usual.  The GEMM therefore
// runs while the layer is still arriving, no SM is given up to communication, and when the kernel ends the whole layer
// buffer is gathered for the GEMMs that follow.
//
// scatter (GEMM -> reduce-scatter, MODE_SCATTER): the fp32 epilogue does not store C locally; every row piece goes to the
// rank that owns its position of the flat layer gradient, into that owner's slot for this rank (slot r of the owner's
// reduce buffer = contributions of rank r to the owner's shard).  The owner then sums its `world` slots locally in rank
// order.
struct FusedArgs {
  // gather
  int gather;
  int world, rank;
  unsigned long long* counters;      // [number of B column blocks] bytes landed, monotonic over calls (device memory of this GPU)
  unsigned long long epoch;          // this call completes a block when its counter reaches epoch * bytes of the block
  const void* peer_in[MAX_RANKS];
  uint8_t* layer_buf;
  long long shard_bytes, b_byte_off;
  // optional: sum of squares of the (alpha-scaled) fp32 output, atomically added to *sumsq (gradient-norm fusion)
  float* sumsq;
  // scatter
  int scatter;
  int wire_bf16;                     // the slots hold bf16 (the owner accumulates in fp32); else fp32
  void* peer_grad[MAX_RANKS];
  long long c_flat_off, shard_numel;
};

YF_DEVINL unsigned long long ld_relaxed_gpu_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
YF_DEVINL void red_add_relaxed_gpu_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.relaxed.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// counters of split tiles: has every other range arrived / arrive (true: as the last one)
YF_DEVINL bool split_others_arrived(unsigned long long* ctr, unsigned long long nonce, int splits) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(ctr) : "memory");
  return v == ((nonce << 8) | (unsigned long long)(splits - 1));
}
YF_DEVINL bool split_arrive(unsigned long long* ctr, unsigned long long nonce, int splits) {
  unsigned long long old = ld_relaxed_gpu_u64(ctr);
  for (;;) {  // ends: a failed exchange means that another range of the tile has arrived
    const unsigned long long n = ((old >> 8) == nonce ? (old & 255ull) : 0ull) + 1ull;
    const unsigned long long seen = atomicCAS(ctr, old, (nonce << 8) | n);
    if (seen == old) return n == (unsigned long long)splits;
    old = seen;
  }
}
YF_DEVINL void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

YF_DEVINL void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)),
               "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
YF_DEVINL void bulk_store(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(reinterpret_cast<uint64_t>(gdst)),
               "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
YF_DEVINL void tma_store_wait1() { asm volatile("cp.async.bulk.wait_group 1;" ::: "memory"); }

// Communication role of the gather mode: ONE thread of every CTA.  Piece q of the layer (q = 0, 1, ...) is piece q / world
// of the shard of rank (rank + q % world) % world, so consecutive pieces come from different owners and, at any moment, the
// ranks read from different peers; CTA c moves the pieces c, c + grid, c + 2 grid, ...  A piece goes peer -> ring slot
// (bulk load, completion on an mbarrier) -> local layer buffer (bulk store); four loads and two stores are in flight.
constexpr int COMM_PIECE = 16384;
constexpr int COMM_SLOTS = 6;
constexpr int COMM_AHEAD = 4;   // loads in flight per CTA (64 KB; x 148 CTAs covers the NVLink bandwidth-delay product with margin)

__device__ void gather_comm_role(const FusedArgs& fa, long long b_bytes, long long block_bytes, uint8_t* ring, uint64_t* ring_bars) {
  const long long pps = (fa.shard_bytes + COMM_PIECE - 1) / COMM_PIECE;  // pieces per shard
  const long long total = pps * fa.world;
  const long long first = blockIdx.x, step = gridDim.x;
  const long long mine = first < total ? (total - first + step - 1) / step : 0;
  auto piece = [&](long long i, const uint8_t*& src, long long& layer_off, uint32_t& bytes) {
    const long long q = first + i * step;
    const int owner = (fa.rank + (int)(q % fa.world)) % fa.world;
    const long long lo = (q / fa.world) * COMM_PIECE;
    bytes = (uint32_t)min((long long)COMM_PIECE, fa.shard_bytes - lo);
    src = reinterpret_cast<const uint8_t*>(fa.peer_in[owner]) + lo;
    layer_off = (long long)owner * fa.shard_bytes + lo;
  };
  auto issue_load = [&](long long i) {
    const uint8_t* src; long long off; uint32_t bytes;
    piece(i, src, off, bytes);
    const int slot = (int)(i % COMM_SLOTS);
    mbar_expect_tx(&ring_bars[slot], bytes);
    bulk_load(ring + slot * COMM_PIECE, src, bytes, &ring_bars[slot]);
  };
  // piece i has been written to the layer buffer: credit the B column blocks it overlaps
  auto publish = [&](long long i) {
    const uint8_t* src; long long off; uint32_t bytes;
    piece(i, src, off, bytes);
    long long lo = max(off, fa.b_byte_off) - fa.b_byte_off, hi = min(off + (long long)bytes, fa.b_byte_off + b_bytes) - fa.b_byte_off;
    if (lo >= hi) return;
    // The piece's bulk store has completed (wait_group): its bytes have been written at the L2, the point where the
    // counter's atomic add is performed too, so the add cannot be seen before them.  No fence here: a release fence or a
    // proxy fence waits for everything this SM has in flight (the GEMM's own loads, stores and MMAs), tens of microseconds
    // per piece while the GEMM runs; the reader acquires and fences once per tile instead.
    while (lo < hi) {
      const long long blk = lo / block_bytes;
      const long long end = min(hi, (blk + 1) * block_bytes);
      red_add_relaxed_gpu_u64(fa.counters + blk, (unsigned long long)(end - lo));
      lo = end;
    }
  };
  for (long long i = 0; i < COMM_AHEAD && i < mine; ++i) issue_load(i);
  long long done = 0, stored = 0;  // pieces published / pieces whose store has been issued
#ifdef YF_GATHER_PROFILE
  unsigned long long tp[5] = {0, 0, 0, 0, 0};
  unsigned long long t_a = yf_globaltimer(), t_b;
#define YF_TICK(k) t_b = yf_globaltimer(); tp[k] += t_b - t_a; t_a = t_b;
#else
#define YF_TICK(k)
#endif
  for (long long i = 0; i < mine; ++i, ++stored) {
    const int slot = (int)(i % COMM_SLOTS);
    if (!mbar_wait(&ring_bars[slot], (uint32_t)((i / COMM_SLOTS) & 1), 12)) break;  // gave up: nothing more is copied or published
    YF_TICK(0)
    const uint8_t* src; long long off; uint32_t bytes;
    piece(i, src, off, bytes);
    bulk_store(fa.layer_buf + off, ring + slot * COMM_PIECE, bytes);
    tma_store_commit();
    tma_store_wait_read1();  // every store but this one has finished reading its slot: the slot of piece i - 2 is free
    YF_TICK(1)
    if (i + COMM_AHEAD < mine) issue_load(i + COMM_AHEAD);  // into slot (i + 4) % 6 == (i - 2) % 6
    YF_TICK(2)
    tma_store_wait1();       // every store but this one has completed: piece i - 1 is in the layer buffer
    YF_TICK(3)
    if (i >= 1) { publish(i - 1); done = i; }
    YF_TICK(4)
  }
#ifdef YF_GATHER_PROFILE
  for (int k = 0; k < 5; ++k) fa.counters[1024 + 8 * blockIdx.x + k] = tp[k];
  fa.counters[1024 + 8 * blockIdx.x + 5] = (unsigned long long)mine;
#endif
  tma_store_wait0();
  for (long long i = done; i < stored; ++i) publish(i);
}

// 128 registers a thread, 28 672 of the SM's 65 536: blocks of the pull reduce-scatter (64 registers) and of AdamW find room next to a
// persistent CTA.  The split instantiations spill 120 to 132 bytes for it, the SwiGLU one 12, around their epilogues.
template <int BLOCK_N, int CG, int MODE>
__global__ void __maxnreg__(128)
gemm_bf16_tcgen05_kernel(const __grid_constant__ GroupMaps maps, const __grid_constant__ CUtensorMap tma_c, GemmArgs args, FusedArgs fa) {
  using Cfg = GemmCfg<BLOCK_N, CG, MODE>;
  // CG == 2: the grid is a sequence of CTA pairs (clusters of two); a pair works on one 256 x BLOCK_N tile, CTA `crank` of
  // the pair on its rows [crank * 128, +128) with the B rows [crank * BLOCK_N / 2, +BLOCK_N / 2) in its shared memory
  const uint32_t crank = (CG == 2) ? cluster_ctarank() : 0u;
  const bool leader = crank == 0;
  const int unit = (int)blockIdx.x / CG;        // index among the tile workers (CTAs or pairs)
  const int nunits = (int)gridDim.x / CG;
  constexpr int STAGES = Cfg::STAGES;
  constexpr int TILE_M = BLOCK_M * CG;
  constexpr int B_ROWS = Cfg::B_ROWS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + STAGES * Cfg::STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + Cfg::STAGING_BYTES);
  uint64_t* full = bars;                 // [STAGES]  (pairs: only the leader's are used, both CTAs' loads count there)
  uint64_t* empty = bars + STAGES;       // [STAGES]
  uint64_t* tfull = bars + 2 * STAGES;   // [2]
  uint64_t* tempty = tfull + 2;          // [2]       (pairs: only the leader's are used)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  uint64_t* ring_bars = reinterpret_cast<uint64_t*>(tmem_slot + 2);   // [COMM_SLOTS], gather mode
  uint8_t* ring = staging + Cfg::STAGING_BYTES - Cfg::RING_BYTES;     // gather mode: the tail of the staging area

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int K = args.K;
  const int num_m = (args.M + TILE_M - 1) / TILE_M;
  const int bn = MODE == MODE_SWAP ? args.bn : BLOCK_N;
  const int num_n = (args.N + bn - 1) / bn;
  const int num_k = (K + BLOCK_K - 1) / BLOCK_K;
  const bool grouped = (MODE == MODE_SCATTER) && args.n_prob > 0;
  const int num_tiles = grouped ? args.steps : num_m * num_n;  // steps of the tile loop (a grouped step may be empty)
  const int num_items = num_tiles + (MODE == MODE_SPLIT ? args.split_tiles * (args.splits - 1) : 0);
  constexpr int GROUP_M = 16 / CG;  // 2048 rows of A share a column block of B through L2

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&maps.a[0]);
    tma_prefetch_desc(&maps.b[0]);
    tma_prefetch_desc(&tma_c);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 4 * CG);  // one arrival per epilogue warp of every CTA of the pair
    }
    if (MODE == MODE_GATHER)
      for (int i = 0; i < COMM_SLOTS; ++i) mbar_init(&ring_bars[i], 1);
    mbar_fence_init();
  }
  if (warp == 1) {
    if (CG == 2) {
      tmem_alloc_pair(tmem_slot, Cfg::TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync_all();  // the peer's barriers and TMEM exist before anything is sent to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // step t of this launch -> problem p, first row m0 (of this CTA) and first column n0 of the tile; false: empty step
  auto tile_coords = [&](int t, int& p, int& m0, int& n0) -> bool {
    if (grouped) {
      const int o = (fa.rank + 1 + t % fa.world) % fa.world;
      const int g = args.own_start[o] + t / fa.world;
      if (g >= args.own_start[o + 1]) return false;  // this owner has fewer tiles than the largest one
      p = 0;
      while (p + 1 < args.n_prob && g >= args.tile_prefix[p + 1]) ++p;
      const int local = g - args.tile_prefix[p];
      const int nn = (args.Np[p] + BLOCK_N - 1) / BLOCK_N;
      m0 = (local / nn) * TILE_M + (int)crank * BLOCK_M;
      n0 = (local % nn) * BLOCK_N;
      return true;
    }
    p = 0;
    const int per_group = GROUP_M * num_n;
    const int g = t / per_group;
    const int first_m = g * GROUP_M;
    const int gsize = min(GROUP_M, num_m - first_m);
    const int r = t - g * per_group;
    m0 = (first_m + r % gsize) * TILE_M + (int)crank * BLOCK_M;
    n0 = (r / gsize) * bn;
    return true;
  };

  if (warp == 0 || (is_plain(MODE) && warp == 6)) {
    // ------------------------------------------------------------ TMA producers
    // Plain mode has two producers that take turns: waiting, announcing the bytes and issuing the copies of a K block cost
    // one thread about 190 ns, which is more than the MMAs of a narrow tile take.  The number of stages is even, so
    // producer j fills the stages of its parity.
    constexpr int PRODUCERS = is_plain(MODE) ? 2 : 1;
    static_assert(STAGES % PRODUCERS == 0 || PRODUCERS == 1, "every producer has its own stages");
    const int producer = warp == 0 ? 0 : 1;
    if (elect_one()) {
      uint32_t s = producer, ph = 0;  // ring position: stage and how often (mod 2) the ring has gone round
      int skip = producer;            // K blocks in front of this producer's next one
      const uint32_t full_leader = CG == 2 ? mapa_shared(smem_u32(full), 0) : 0u;
      bool alive = true;
      for (int t = unit; t < num_items && alive; t += nunits) {
        const WorkItem w = work_item<MODE>(args, t, num_k);
        int p, m0, n0;
        if (!tile_coords(w.tile, p, m0, n0)) continue;
        const CUtensorMap* tma_a = &maps.a[p];
        const CUtensorMap* tma_b = &maps.b[p];
        // the weight may lie in pieces: B, or A in the swapped form; w_at: first row of the current one
        constexpr bool SWAP = MODE == MODE_SWAP;
        const bool w_mn = SWAP ? args.a_mn : args.b_mn;
        int w_at = 0;
        auto next_piece = [&](int i) {
          w_at = args.parts[i];
          if (SWAP) tma_a = &maps.a[i + 1];
          else tma_b = &maps.b[i + 1];
        };
        if (is_plain(MODE) && args.n_parts > 1 && !w_mn)
          for (int i = 0; (SWAP ? m0 : n0) >= args.parts[i]; ++i) next_piece(i);
        const int N = grouped ? args.Np[p] : args.N;
        if (MODE == MODE_GATHER) {
          // the rows [n0, n0 + BLOCK_N) of B must have landed in the local layer buffer: the column block's counter says so
          const int blk = n0 / BLOCK_N;
          const unsigned long long want = fa.epoch * (unsigned long long)((long long)min(BLOCK_N, N - n0) * K * 2);
          // Poll with relaxed loads and pauses: an acquire per poll is a memory fence per poll, and such a fence waits for
          // everything the busy SM has in flight (tens of microseconds) and holds up the communication warp next door.
          // The rows were written by bulk stores (asynchronous proxy) of CTAs of this GPU and are read by TMA (the same
          // proxy) straight from the L2, where they were complete before the counter moved; the TMA loads are issued after
          // the poll has returned.  So no acquire and no proxy fence follow: either one waits for the communication warp's
          // copies in flight, which never pause (measured: 1.7 ms instead of 0.34 ms for the kernel).
          const uint64_t t0 = yf_globaltimer();
          for (uint32_t spin = 0; ld_relaxed_gpu_u64(fa.counters + blk) < want; ++spin) {
            __nanosleep(400);
            if ((spin & 63u) == 63u && (yf_aborted() || yf_globaltimer() - t0 > YF_WAIT_NS_DEFAULT)) {
              yf_raise(YF_ERR_FLAG_TIMEOUT, 11);
              alive = false;
              break;
            }
          }
          if (!alive) break;
        }
        int nb = n0 + (int)crank * (SWAP ? bn / 2 : B_ROWS) - (!SWAP && !args.b_mn ? w_at : 0);  // first B row this CTA holds
        const int ma = m0 - (SWAP && !args.a_mn ? w_at : 0);
        const uint32_t stage_tx = SWAP ? Cfg::A_BYTES + bn / 2 * (BLOCK_K * 2) : Cfg::STAGE_BYTES;  // bytes that land in a CTA's stage
        if (MODE == MODE_SWIGLU) {  // a pair: its leader holds gate rows, the other CTA the same rows of up
          nb = n0 / 2;
          tma_b = &maps.b[crank];
        }
        const bool k_parts = is_plain(MODE) && args.n_parts > 1 && w_mn;
        int piece = 0;
        int kb = w.kb0 + skip;
        for (; kb < w.kb1; kb += PRODUCERS) {
          if (k_parts)
            while (kb * BLOCK_K >= args.parts[piece]) next_piece(piece++);
          if (!mbar_wait(&empty[s], ph ^ 1, 10)) { alive = false; break; }
          uint8_t* sa = smem + s * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + Cfg::A_BYTES;
          const int k0 = kb * BLOCK_K, ka0 = SWAP && args.a_mn ? k0 - w_at : k0, kb0 = !SWAP && args.b_mn ? k0 - w_at : k0;
          if (CG == 2) {
            // both CTAs' bytes are counted on the leader's barrier (the thread that issues the MMAs waits there)
            if (leader) mbar_expect_tx(&full[s], 2 * stage_tx);
            const uint32_t fb = full_leader + s * 8;
            if (!args.a_mn) {
              tma_load_2d_pair(sa, tma_a, fb, ka0, ma);
            } else {
#pragma unroll
              for (int j = 0; j < BLOCK_M / 64; ++j) tma_load_2d_pair(sa + j * (BLOCK_K * 128), tma_a, fb, ma + j * 64, ka0);
            }
            if (!args.b_mn) {
              tma_load_2d_pair(sb, tma_b, fb, kb0, nb);
            } else {
#pragma unroll
              for (int j = 0; j < B_ROWS / 64; ++j) tma_load_2d_pair(sb + j * (BLOCK_K * 128), tma_b, fb, nb + j * 64, kb0);
            }
          } else {
            mbar_expect_tx(&full[s], stage_tx);
            if (!args.a_mn) {
              tma_load_2d(sa, tma_a, &full[s], ka0, ma);
            } else {
#pragma unroll
              for (int j = 0; j < BLOCK_M / 64; ++j) tma_load_2d(sa + j * (BLOCK_K * 128), tma_a, &full[s], ma + j * 64, ka0);
            }
            if (!args.b_mn) {
              tma_load_2d(sb, tma_b, &full[s], kb0, nb);
            } else {
#pragma unroll
              for (int j = 0; j < B_ROWS / 64; ++j) tma_load_2d(sb + j * (BLOCK_K * 128), tma_b, &full[s], nb + j * 64, kb0);
            }
          }
          s += PRODUCERS;
          if (s >= STAGES) { s -= STAGES; ph ^= 1; }
        }
        skip = kb - w.kb1;
      }
      if (!alive) {
        // give copies already in flight a bounded time to land before the CTA may exit
        const uint64_t t0 = yf_globaltimer();
        while (yf_globaltimer() - t0 < 200000ull) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (pairs: the leader CTA issues for both)
    if (leader && elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(TILE_M, bn, args.a_mn, args.b_mn);
      // Shared-memory descriptors: the upper words are constants, the lower ones advance by the stage and the K step (in
      // units of 16 bytes; the whole of shared memory fits the address field).  One thread issues everything: what it
      // computes per K block has to stay below the 256 to 512 cycles that the block's MMAs take.
      const uint64_t a0 = umma_smem_desc_sw128(smem_u32(smem), args.a_mn ? BLOCK_K * 128 : 0, 1024);
      const uint64_t b0 = umma_smem_desc_sw128(smem_u32(smem) + Cfg::A_BYTES, args.b_mn ? BLOCK_K * 128 : 0, 1024);
      const uint32_t a_kstep = (args.a_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4, b_kstep = (args.b_mn ? UMMA_K * 128 : UMMA_K * 2) >> 4;
      const uint32_t empty_0 = CG == 2 ? mapa_shared(smem_u32(empty), 0) : 0u, empty_1 = CG == 2 ? mapa_shared(smem_u32(empty), 1) : 0u;
      uint32_t s = 0, ph = 0;
      bool alive = true;
      int lt = 0;
      for (int t = unit; t < num_items && alive; t += nunits) {
        const WorkItem w = work_item<MODE>(args, t, num_k);
        {
          int p, m0, n0;
          if (!tile_coords(w.tile, p, m0, n0)) continue;
        }
        const int acc = lt & 1;
        const uint32_t acc_ph = (lt >> 1) & 1;
        ++lt;
        if (!mbar_wait(&tempty[acc], acc_ph ^ 1, 20)) { alive = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BLOCK_N;
        uint32_t add = 0;  // the first MMA of an item overwrites the accumulator
        for (int kb = w.kb0; kb < w.kb1; ++kb) {
          if (!mbar_wait(&full[s], ph, 21)) { alive = false; break; }
          tc_fence_after();
          const uint64_t a_desc = a0 + s * (Cfg::STAGE_BYTES >> 4), b_desc = b0 + s * (Cfg::STAGE_BYTES >> 4);
#pragma unroll
          for (int k = 0; k < BLOCK_K / UMMA_K; ++k) {
            if (CG == 2) tc_mma_bf16_pair(d_tmem, a_desc + k * a_kstep, b_desc + k * b_kstep, idesc, add);
            else tc_mma_bf16(d_tmem, a_desc + k * a_kstep, b_desc + k * b_kstep, idesc, add);
            add = 1;
          }
          // frees the stage (in both CTAs of a pair) once these MMAs have read it
          if (CG == 2) {
            tc_commit_pair(empty_0 + s * 8);
            tc_commit_pair(empty_1 + s * 8);
          } else {
            tc_commit(&empty[s]);
          }
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (alive) {
          if (CG == 2) {
            const uint32_t tb = smem_u32(&tfull[acc]);
            tc_commit_pair(mapa_shared(tb, 0));
            tc_commit_pair(mapa_shared(tb, 1));
          } else {
            tc_commit(&tfull[acc]);
          }
        }
      }
    }
  } else if (MODE == MODE_GATHER && warp == 6) {
    // ------------------------------------------------------------ communication role (gather mode)
    if (lane == 0) gather_comm_role(fa, (long long)args.N * K * 2, (long long)BLOCK_N * K * 2, ring, ring_bars);
  } else {
    // ------------------------------------------------------------ epilogue (4 warps = 128 TMEM lanes)
    // TMEM -> registers -> 128-byte-swizzled staging block in shared memory -> TMA store (or TMA
    // reduce-add when accumulating): full 128-byte lines leave the SM, edges are clipped by the TMA unit.
    // Every warp stages and stores its own 32 rows (two blocks of [32 rows x 128 bytes]), so the four warps run without
    // barriers between them and hide each other's latencies.
    const int q = warp & 3;  // a warp may only touch TMEM lanes [32*(warp%4), +32)
    const int r_in_tile = q * 32 + lane;
    const bool store_thread = (threadIdx.x == 64);
    const int cols_per_chunk = args.out_f32 ? 32 : 64;
    const int n_chunks = BLOCK_N / cols_per_chunk;
    bool alive = true;
    int lt = 0;
    uint32_t chunk_ctr = 0;
    float ss = 0.f;  // sum of squares of this thread's outputs (rows / columns past the edges are exact zeros)
    for (int t = unit; t < num_items && alive; t += nunits) {
      const WorkItem w = work_item<MODE>(args, t, num_k);
      int p, m0, n0;
      if (!tile_coords(w.tile, p, m0, n0)) continue;
      const int M = grouped ? args.Mp[p] : args.M, N = grouped ? args.Np[p] : args.N;
      const long long c_flat_off = grouped ? args.flat_off[p] : fa.c_flat_off;
      const int acc = lt & 1;
      const uint32_t acc_ph = (lt >> 1) & 1;
      ++lt;
      const bool gave_up = !mbar_wait(&tfull[acc], acc_ph, 30);
      if (MODE == MODE_SCATTER) {
        if (!__all_sync(0xffffffffu, !gave_up)) { alive = false; break; }  // per-warp epilogue: a warp leaves as a whole
      } else if (named_bar_or(1, 128, gave_up)) {  // the four warps share named barriers below: they leave together
        alive = false;
        break;
      }
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BLOCK_N;
      const float alpha = alpha_of(args);
      if constexpr (MODE == MODE_SCATTER) {
        // GEMM -> reduce-scatter.  Every thread owns one row of the accumulator: it moves 64 columns at a time from its
        // TMEM lane into its own row of a staging block and sends that 256-byte piece with one bulk store (two where the
        // piece straddles a shard boundary) to the slot that the owning rank keeps for this rank.  No thread touches
        // another thread's row, so the epilogue needs no block-level barrier; bulk groups are per thread.
        // Wire format fp32 (64 columns per piece) or bf16 (128 columns per piece; the owner still accumulates in fp32).
        const int m = m0 + r_in_tile;
        const int esz = fa.wire_bf16 ? 2 : 4;
        const int piece_cols = fa.wire_bf16 ? 2 * SCATTER_COLS : SCATTER_COLS;
        const int n_pieces = BLOCK_N / piece_cols;
        const long long align_mask = fa.wire_bf16 ? 7 : 3;  // 16-byte pieces
#pragma unroll 1
        for (int c = 0; c < n_pieces; ++c, ++chunk_ctr) {
          uint8_t* srow = staging + (chunk_ctr & 1) * (BLOCK_M * SCATTER_PITCH) + r_in_tile * SCATTER_PITCH;
          tma_store_wait_read1();  // the store that read this row two pieces ago has finished reading
          if (fa.wire_bf16) {
#pragma unroll
            for (int quarter = 0; quarter < 4; ++quarter) {
              uint32_t r[32];
              tmem_ld32(taddr + c * piece_cols + quarter * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                uint4 o;
                o.x = pack_bf16x2(alpha * __uint_as_float(r[8 * j + 0]), alpha * __uint_as_float(r[8 * j + 1]));
                o.y = pack_bf16x2(alpha * __uint_as_float(r[8 * j + 2]), alpha * __uint_as_float(r[8 * j + 3]));
                o.z = pack_bf16x2(alpha * __uint_as_float(r[8 * j + 4]), alpha * __uint_as_float(r[8 * j + 5]));
                o.w = pack_bf16x2(alpha * __uint_as_float(r[8 * j + 6]), alpha * __uint_as_float(r[8 * j + 7]));
                *reinterpret_cast<uint4*>(srow + quarter * 64 + j * 16) = o;
              }
            }
          } else {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              uint32_t r[32];
              tmem_ld32(taddr + c * piece_cols + half * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                float4 o;
                o.x = alpha * __uint_as_float(r[4 * j + 0]);
                o.y = alpha * __uint_as_float(r[4 * j + 1]);
                o.z = alpha * __uint_as_float(r[4 * j + 2]);
                o.w = alpha * __uint_as_float(r[4 * j + 3]);
                *reinterpret_cast<float4*>(srow + half * 128 + j * 16) = o;
              }
            }
          }
          if (c == n_pieces - 1) {  // accumulator fully read: hand it back to the MMA warp (of the leader CTA)
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              if (CG == 2) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[acc]), 0));
              else mbar_arrive(&tempty[acc]);
            }
          }
          fence_proxy_async_smem();
          const int col = n0 + c * piece_cols;
          if (m < M && col < N) {
            const long long ncols = min(piece_cols, N - col);
            const long long f = c_flat_off + (long long)m * N + col;      // position in the flat layer gradient
            const long long o = f / fa.shard_numel;                       // owner rank
            const long long loc = f - o * fa.shard_numel;
            const long long first = min(ncols, fa.shard_numel - loc);
#ifdef YF_DEBUG_BOUNDS
            // debug build: a piece that would leave the owners' slots is recorded and skipped instead of stored
            if (f < 0 || o >= fa.world || (first < ncols && o + 1 >= fa.world) || loc < 0 || (first & align_mask) || (loc & align_mask)) {
              yf_raise(YF_ERR_BAD_ARGUMENT, 40);
              tma_store_commit();
              continue;
            }
#endif
            (void)align_mask;
            uint8_t* dst = reinterpret_cast<uint8_t*>(fa.peer_grad[o]) + ((long long)fa.rank * fa.shard_numel + loc) * esz;
            bulk_store(dst, srow, (uint32_t)(first * esz));
            if (first < ncols) {
              uint8_t* dst2 = reinterpret_cast<uint8_t*>(fa.peer_grad[o + 1]) + (long long)fa.rank * fa.shard_numel * esz;
              bulk_store(dst2, srow + first * esz, (uint32_t)((ncols - first) * esz));
            }
          }
          tma_store_commit();
        }
      } else {
      auto free_accumulator = [&]() {  // fully read: hand it back to the MMA warp (of the leader CTA)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (CG == 2) mbar_arrive_cluster(mapa_shared(smem_u32(&tempty[acc]), 0));
          else mbar_arrive(&tempty[acc]);
        }
      };
      // One range of a split tile: its sums go to its slot unless all other ranges are there already.  A slot holds float4
      // column groups of 128 rows (512 contiguous bytes per warp and access).  The last range adds the others to its
      // accumulator, in the order of the ranges, and carries on with the output as for a whole tile.
      if (MODE == MODE_SPLIT && w.part >= 0) {
        const bool rows_here = m0 + q * 32 < M;  // this warp's rows
        const int cta_tile = w.tile * CG + (int)crank;
        unsigned long long* ctr = args.counters + cta_tile;
        float4* slot0 = reinterpret_cast<float4*>(args.slots) + (long long)cta_tile * args.splits * (BLOCK_M * BLOCK_N / 4) + r_in_tile;
        bool last = named_bar_or(1, 128, store_thread && split_others_arrived(ctr, args.nonce, args.splits));
        if (!last) {
          float4* mine = slot0 + w.part * (BLOCK_M * BLOCK_N / 4);
#pragma unroll 1
          for (int c = 0; c < BLOCK_N / 32; ++c) {
            uint32_t r[32];
            tmem_ld32(taddr + c * 32, r);
            tmem_ld_wait();
            if (rows_here) {
#pragma unroll
              for (int j = 0; j < 8; ++j)
                __stcg(mine + (c * 8 + j) * BLOCK_M, make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                                                 __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3])));
            }
          }
          named_bar_sync(1, 128);  // all 128 threads' sums are written before one of them publishes
          if (store_thread) {
            __threadfence();
            last = split_arrive(ctr, args.nonce, args.splits);
            __threadfence();
          }
          last = named_bar_or(1, 128, store_thread && last);
        }
        if (!last) {
          free_accumulator();
          continue;
        }
        if (store_thread) *ctr = 0ull;
        // three 32-column pieces of other ranges in flight: of one block of columns, or with one other range of three blocks
        const int others = args.splits - 1;
        const int step = others == 1 ? 3 : 1;
#pragma unroll 1
        for (int c = 0; c < BLOCK_N / 32; c += step) {
          float4 x[3][8];
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            const int range = others == 1 ? 1 - w.part : i + (i >= w.part ? 1 : 0), block = others == 1 ? c + i : c;
            const bool there = rows_here && (others == 1 ? block < BLOCK_N / 32 : i < others);
            const float4* src = slot0 + range * (BLOCK_M * BLOCK_N / 4) + block * 8 * BLOCK_M;
#pragma unroll
            for (int j = 0; j < 8; ++j) x[i][j] = there ? __ldcg(src + j * BLOCK_M) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int b = 0; b < 3; ++b) {
            if (b >= step || c + b >= BLOCK_N / 32) break;
            uint32_t r[32];
            tmem_ld32(taddr + (c + b) * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float own = __uint_as_float(r[j]);
              auto at = [&](int i) { return (j & 3) == 0 ? x[i][j / 4].x : (j & 3) == 1 ? x[i][j / 4].y : (j & 3) == 2 ? x[i][j / 4].z : x[i][j / 4].w; };
              float sum;
              if (b > 0 || others == 1) {
                sum = own + at(b);  // two terms: the same sum in either order
              } else {  // in the order of the ranges, the own one is number w.part
                sum = w.part == 0 ? own + at(0) : at(0) + (w.part == 1 ? own : at(1));
                sum += w.part <= 1 ? at(1) : (w.part == 2 ? own : at(2));
                sum += w.part <= 2 ? at(2) : own;
              }
              r[j] = __float_as_uint(sum);
            }
            tmem_st32(taddr + (c + b) * 32, r);
          }
        }
        tmem_st_wait();
      }
      if constexpr (MODE == MODE_SWAP) {
        // a thread owns an output column (weight row), TMEM columns are tokens: 32 tokens at a time through a block of
        // [32 tokens x 32 columns] bf16 (a warp's stores fill one 64-byte row each), two TMA stores of 16 tokens
        const int col = m0 + r_in_tile;
#pragma unroll 1
        for (int c = 0; c < bn; c += 32, ++chunk_ctr) {
          uint8_t* stg = staging + q * 8192 + (chunk_ctr & 3) * 2048;
          if (lane == 0) tma_store_wait_read3();  // the stores that last read this block have finished reading
          __syncwarp();
          unsigned short res[32];
          if (args.R != nullptr) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              res[j] = col < M && n0 + c + j < N ? __ldg(static_cast<const unsigned short*>(args.R) + (long long)(n0 + c + j) * args.ldr + col) : 0;
          }
          uint32_t r[32];
          tmem_ld32(taddr + c, r);
          tmem_ld_wait();
          if (c + 32 >= bn) free_accumulator();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            float v = alpha * __uint_as_float(r[j]);
            if (args.R != nullptr) v = fmaf(alpha, __uint_as_float(r[j]), __uint_as_float((uint32_t)res[j] << 16));
            *reinterpret_cast<__nv_bfloat16*>(stg + j * 64 + lane * 2) = __float2bfloat16_rn(v);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int x = m0 + q * 32;
            if (x < M && n0 + c < N) tma_store_2d(&tma_c, stg, x, n0 + c);
            if (x < M && c + 16 < bn && n0 + c + 16 < N) tma_store_2d(&tma_c, stg + 1024, x, n0 + c + 16);
            tma_store_commit();
          }
        }
        continue;
      }
      if constexpr (MODE == MODE_SWIGLU) {
        // 64 columns of one output: 32 packed pairs of this thread's row -> this warp's staging block -> TMA store
        auto store64 = [&](const CUtensorMap* map, int x, const uint32_t (&v)[32]) {  // (F is a multiple of a tile's 128)
          uint8_t* stg = staging + q * 8192 + (chunk_ctr & 1) * 4096;
          ++chunk_ctr;
          if (lane == 0) tma_store_wait_read1();
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<uint4*>(stg + lane * 128 + ((j ^ (lane & 7)) << 4)) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            const int y = m0 + q * 32;
            if (y < M) tma_store_2d(map, stg, x, y);
            tma_store_commit();
          }
        };
        auto load64 = [&](int col, uint32_t (&v)[32]) {  // 64 accumulator columns of this thread's row, rounded to bf16
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t r[32];
            tmem_ld32(taddr + col + half * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) v[half * 16 + j] = pack_bf16x2(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          }
        };
        const int F = N / 2;
#pragma unroll 1
        for (int c = 0; c < 2; ++c) {
          const int x = n0 / 2 + c * 64;
          uint32_t g[32], u[32];
          load64(c * 64, g);
          if (args.store_gu) store64(&tma_c, x, g);
          load64(128 + c * 64, u);
          if (c == 1) free_accumulator();
          if (args.store_gu) store64(&tma_c, F + x, u);
          if (m0 + r_in_tile < M) {  // rows past the end are zeros, and 0 / x takes the long way through the division
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              const float2 gf = unpack_bf16x2(g[j]), uf = unpack_bf16x2(u[j]);
              g[j] = pack_bf16x2(gf.x / (1.f + __expf(-gf.x)) * uf.x, gf.y / (1.f + __expf(-gf.y)) * uf.y);
            }
          }
          store64(&maps.a[1], x, g);
        }
        continue;
      }
#pragma unroll 1
      for (int c = 0; c < n_chunks; ++c, ++chunk_ctr) {
        uint8_t* stg = staging + q * 8192 + (chunk_ctr & 1) * 4096;
        uint8_t* srow = stg + lane * 128;
        if (lane == 0) tma_store_wait_read1();  // the store that last read this block has finished reading
        __syncwarp();
        if (args.out_f32) {
          uint32_t r[32];
          tmem_ld32(taddr + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 o;
            o.x = alpha * __uint_as_float(r[4 * j + 0]);
            o.y = alpha * __uint_as_float(r[4 * j + 1]);
            o.z = alpha * __uint_as_float(r[4 * j + 2]);
            o.w = alpha * __uint_as_float(r[4 * j + 3]);
            ss += o.x * o.x + o.y * o.y + o.z * o.z + o.w * o.w;
            *reinterpret_cast<float4*>(srow + ((j ^ (lane & 7)) << 4)) = o;
          }
        } else {
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            // the residual of this thread's row: 4 x 16 bytes, requested before the accumulator is read (N % 8 == 0)
            uint4 res[4] = {};
            if (args.R != nullptr) {
              const int row = m0 + r_in_tile, col = n0 + c * 64 + half * 32;
              if (row < M) {
                const uint4* rp = reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(args.R) + (long long)row * args.ldr + col);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                  if (col + 8 * j < N) res[j] = __ldg(rp + j);
              }
            }
            uint32_t r[32];
            tmem_ld32(taddr + c * 64 + half * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint32_t rw[4] = {res[j].x, res[j].y, res[j].z, res[j].w};
              uint32_t ow[4];
#pragma unroll
              for (int w = 0; w < 4; ++w)  // a bf16 pair: low half = even column
                ow[w] = pack_bf16x2(fmaf(alpha, __uint_as_float(r[8 * j + 2 * w]), __uint_as_float(rw[w] << 16)),
                                    fmaf(alpha, __uint_as_float(r[8 * j + 2 * w + 1]), __uint_as_float(rw[w] & 0xffff0000u)));
              *reinterpret_cast<uint4*>(srow + (((half * 4 + j) ^ (lane & 7)) << 4)) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
            }
          }
        }
        if (c == n_chunks - 1) free_accumulator();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int x = n0 + c * cols_per_chunk, y = m0 + q * 32;
          if (x < N && y < M) {
            if (args.accumulate) tma_reduce_add_2d(&tma_c, stg, x, y);
            else tma_store_2d(&tma_c, stg, x, y);
          }
          tma_store_commit();
        }
      }
      }
    }
    if (MODE == MODE_SCATTER || lane == 0) tma_store_wait0();  // all of this thread's stores have completed
    if (fa.sumsq != nullptr) {
      ss = warp_sum(ss);
      if (lane == 0) atomicAdd(fa.sumsq, ss);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync_all();  // neither CTA leaves while the other may still read its shared memory or signal its barriers
  if (warp == 1) {
    tc_fence_after();
    if (CG == 2) tmem_dealloc_pair(tmem_base, Cfg::TMEM_COLS);
    else tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// cudaFuncSetAttribute is per device: remember which devices have the opt-in to large dynamic shared memory
template <typename KernelT>
int ensure_smem_optin(KernelT kernel, int bytes, bool (&done)[64]) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  if (!done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return -(int)e;
    done[dev] = true;
  }
  return 0;
}

// One problem's operands (a grouped launch passes several); for B in pieces: N or K is that of the piece.
struct Operands {
  const void* A;
  const void* B;
  long long lda, ldb;
  int M, N;
  int K;
};

template <int BLOCK_N, int CG, int MODE = MODE_PLAIN>
int launch_gemm(const Operands* ops, int n_ops, GemmArgs args, const FusedArgs& fa, int sm_limit, cudaStream_t stream) {
  // args.splits > 1: the caller's plan (tile shape, whole tiles, workspace) was made for this very configuration
  using Cfg = GemmCfg<BLOCK_N, CG, MODE>;
  if (n_ops < 1 || n_ops > MAX_GROUP) return -1;
  GroupMaps maps;
  memset(&maps, 0, sizeof(maps));
  for (int i = 0; i < n_ops; ++i) {
    const Operands& o = ops[i];
    constexpr bool SWAP = MODE == MODE_SWAP;
    const int ka = SWAP ? o.K : args.K, kb = SWAP ? args.K : o.K, b_rows = SWAP ? args.bn / 2 : Cfg::B_ROWS;
    const CUtensorMap* ma = args.a_mn ? yf_tensor_map_2d(o.A, o.M, ka, o.lda, 64, BLOCK_K, 2, 1)
                                      : yf_tensor_map_2d(o.A, ka, o.M, o.lda, BLOCK_K, BLOCK_M, 2, 1);
    const CUtensorMap* mb = args.b_mn ? yf_tensor_map_2d(o.B, o.N, kb, o.ldb, 64, BLOCK_K, 2, 1)
                                      : yf_tensor_map_2d(o.B, kb, o.N, o.ldb, BLOCK_K, b_rows, 2, 1);
    if (!ma || !mb) return -2;
    maps.a[i] = *ma;
    maps.b[i] = *mb;
  }
  if (MODE == MODE_SWIGLU) {  // the activation's store map
    const CUtensorMap* mact = yf_tensor_map_2d(args.R, args.N / 2, args.M, args.ldr, 64, 32, 2, 1);
    if (!mact) return -2;
    maps.a[1] = *mact;
    n_ops = 2;
  }
  for (int i = n_ops; i < MAX_GROUP; ++i) {  // unused entries hold a valid descriptor all the same
    maps.a[i] = maps.a[0];
    maps.b[i] = maps.b[0];
  }
  const int c_cols = MODE == MODE_SWIGLU && !args.store_gu ? args.N / 2 : args.N;
  const CUtensorMap* mc = MODE == MODE_SWAP ? yf_tensor_map_2d(args.C, args.M, args.N, args.ldc, 32, 16, 2, 0)
                                            : yf_tensor_map_2d(args.C, c_cols, args.M, args.ldc, args.out_f32 ? 32 : 64, 32, args.out_f32 ? 4 : 2, 1);
  if (!mc) return -2;
  static bool optin[64] = {};
  if (int rc = ensure_smem_optin(gemm_bf16_tcgen05_kernel<BLOCK_N, CG, MODE>, Cfg::SMEM_BYTES, optin)) return rc;
  if (int rc = yf_tu_bind_status()) return rc;
  const int tile_m = BLOCK_M * CG;
  int num_tiles = 0;
  if (args.n_prob > 0) {
    for (int i = 0; i < args.n_prob; ++i) {
      args.tile_prefix[i] = num_tiles;
      num_tiles += ((args.Mp[i] + tile_m - 1) / tile_m) * ((args.Np[i] + BLOCK_N - 1) / BLOCK_N);
    }
    args.tile_prefix[args.n_prob] = num_tiles;
    // own_start[o]: first tile (in flat order) whose rows begin in the shard of rank o or later
    int g = 0, o = 0, most = 0;
    args.own_start[0] = 0;
    for (int i = 0; i < args.n_prob; ++i) {
      const int nn = (args.Np[i] + BLOCK_N - 1) / BLOCK_N, nm = (args.Mp[i] + tile_m - 1) / tile_m;
      for (int m = 0; m < nm; ++m, g += nn) {
        const long long owner = (args.flat_off[i] + (long long)m * tile_m * args.Np[i]) / fa.shard_numel;
        while (o < owner && o < fa.world - 1) args.own_start[++o] = g;
      }
    }
    while (o < MAX_RANKS) args.own_start[++o] = num_tiles;
    for (int r = 0; r < fa.world; ++r) most = most > args.own_start[r + 1] - args.own_start[r] ? most : args.own_start[r + 1] - args.own_start[r];
    args.steps = most * fa.world;
    num_tiles = args.steps;
  } else {
    const int bn = MODE == MODE_SWAP ? args.bn : BLOCK_N;
    num_tiles = ((args.M + tile_m - 1) / tile_m) * ((args.N + bn - 1) / bn);
  }
  int sms = yf_num_sms();
  if (sm_limit > 0 && sm_limit < sms) sms = sm_limit;
  int units = sms / CG;
  if (units < 1) return -1;
  // never more CTAs than SMs (producers may wait on other CTAs' communication warps: all of them must be resident); the
  // gather mode keeps every SM's communication warp even when the GEMM has fewer tiles than that
  const int items = num_tiles + (MODE == MODE_SPLIT ? args.split_tiles * (args.splits - 1) : 0);
  if (items < units && MODE != MODE_GATHER) units = items;
  const int grid = units * CG;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3(grid, 1, 1);
  cfg.blockDim = dim3(MODE == MODE_SCATTER ? GEMM_THREADS : WIDE_THREADS, 1, 1);
  cfg.dynamicSmemBytes = Cfg::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CG;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_bf16_tcgen05_kernel<BLOCK_N, CG, MODE>, maps, *mc, args, fa);
  if (e != cudaSuccess) return -(int)e;
  return -(int)cudaGetLastError();
}

template <int BLOCK_N, int CG, int MODE = MODE_PLAIN>
int launch_gemm(const void* A, const void* B, const GemmArgs& args, const FusedArgs& fa, long long lda, long long ldb, int sm_limit,
                cudaStream_t stream) {
  const Operands one = {A, B, lda, ldb, args.M, args.N, args.K};
  return launch_gemm<BLOCK_N, CG, MODE>(&one, 1, args, fa, sm_limit, stream);
}

// ---- plain mode: tile shape and split of the last wave
enum Tile : int { TILE_PAIR256 = 1, TILE_256 = 2, TILE_128 = 3, TILE_64 = 4, TILE_PAIR128 = 5, TILE_SWAP = 6 };
struct Plan {
  int tile, split_tiles, splits, bn;  // bn: tokens per tile of TILE_SWAP
  long long counters, bytes;  // workspace: counters (8 bytes each, rounded up to 256 bytes), then the slots
};
// Per tile shape, measured on one B200 in a stream of launches: us from launch to the end without main loop, and us per K
// block of 64 with all units busy (and, for the wide tiles, the clock that the power cap leaves then).
struct TileShape {
  int cg, bn;
  float fixed_us, kb_us;
};
constexpr TileShape TILE_SHAPES[6] = {{0, 0, 0.f, 0.f}, {2, 256, 7.f, 0.36f}, {1, 256, 6.f, 0.40f}, {1, 128, 4.8f, 0.225f}, {1, 64, 4.2f, 0.155f}, {2, 128, 6.f, 0.20f}};

// What a tile takes whose K blocks take `loop` and whose epilogue takes `epi` us: they overlap, but both move data between the SM and
// the L2.
float tile_time(float loop, float epi) { return loop > epi ? loop + 0.4f * epi : epi + 0.4f * loop; }

// Estimated time of a tile shape and split count.  The epilogue has a fixed part (larger for a pair) and one per column, fp32 or
// bf16; no shape gets more than 5.2 TB/s out of HBM on operands that are read once.  Where K is short (weight gradients of few
// tokens) the fixed part decides, us with tiles of pairs of 256 / 256 / 128 / 64 / pairs of 128 columns (* the choice):
//   fp32 output [57344 x 8192 x 100] 399 / 334* / 363 / 513 / 574, [28672 x 4096 x 333] 146 / 139* / 142 / 163 / 199;
//   bf16 [57344 x 8192 x 100] 307 / 254* / 304 / 383 / 410, [28672 x 4096 x 777] 157* / 173 / 213 / 300 / 213.
// (With an epilogue of 15 and 10.5 ns per column and no fixed part every shape was estimated the same there, and the narrowest won.)
// Splitting: an exchange of partial sums takes 6 to 18 us (a release and an acquire at GPU scope in an SM full of
// asynchronous copies).  Whole tiles behind it hide it, unless a unit gets several ranges one after another.  Long GEMMs
// run against the power cap, where idle units are not all lost, hence the factor of 1.1.
//   [1337 x 4096 x 11008] 139 us whole, 96 us in three ranges; [999 x 5120 x 13824] 142 / 106 us in four;
//   [2048 x 4096 x 22016] 250 / 258 us in four: stays whole.
float plan_us(const TileShape& t, int M, int N, int K, int units, int splits, bool out_f32) {
  const int tile_m = BLOCK_M * t.cg, num_k = (K + BLOCK_K - 1) / BLOCK_K;
  const long long tiles = (long long)((M + tile_m - 1) / tile_m) * ((N + t.bn - 1) / t.bn);
  const long long full = tiles / units, rest = tiles - full * units;
  const float epi = (t.cg == 2 ? 0.95f : 0.39f) + (float)t.bn * (out_f32 ? 0.0118f : 0.0083f);
  const float loop = (float)num_k * t.kb_us, tile_us = tile_time(loop, epi);
  float us = (float)full * tile_us;
  if (rest > 0 && splits == 1) us += tile_us;
  if (rest > 0 && splits > 1) {
    const float rounds = (float)((rest * splits + units - 1) / units), part = loop / (float)splits;
    us += rounds * ((rounds > 1.f && part < 9.f ? 9.f : part) + 4.f) + tile_us - (loop > epi ? loop : epi);
    us *= 1.1f;
  }
  const float exchange_us = rest == 0 || splits == 1 ? 0.f : (full > 0 ? 3.f : 2.f + 4.f * (float)splits);
  const float read_us = ((float)M + (float)N) * (float)K * 2.f / 5.2e6f;
  return t.fixed_us + exchange_us + (us > read_us ? us + 0.1f * read_us : read_us + 0.1f * us);
}

// The swapped form: pairs of 256 weight rows x bn tokens, for every number of token tiles.  A K block takes its MMAs (1.55 ns per
// token with all units busy, a little more than the unswapped form: the epilogue transposes) or its loads (128 + bn / 2 rows at
// 122 GB/s per SM), an epilogue 2 us and 12 ns per token.  Best unswapped / swapped, us:
//   [333 x 27648 x 5120] 98 / 84, [777 x 8192 x 22016] 265 / 218, [777 x 8192 x 8192] 96 / 84, [1337 x 22016 x 4096] 179 / 166,
//   [1337 x 4096 x 4096] 42 / 38; [2048 x 22016 x 4096] 243 / 270 and [999 x 27648 x 5120] 199 / 209 stay unswapped.
float swap_us(int M, int N, int K, int units, int* bn) {
  const int num_k = (K + BLOCK_K - 1) / BLOCK_K, rows = (N + 255) / 256, least = (M + 255) / 256;
  const float read_us = ((float)M + (float)N) * (float)K * 2.f / 5.2e6f;
  float best = 1e30f;
  for (int nt = least; nt < least + 10; ++nt) {
    const int w = ((M + nt - 1) / nt + 15) / 16 * 16;
    if (w > 256 || w < 16) continue;
    const long long tiles = (long long)rows * ((M + w - 1) / w), waves = (tiles + units - 1) / units;
    const float mma = 0.00155f * (float)w, load = (128.f + 0.5f * (float)w) * 0.00105f, loop = (float)num_k * (mma > load ? mma : load);
    const float epi = 2.f + 0.012f * (float)w, us = (float)waves * tile_time(loop, epi);
    const float t = 7.f + (us > read_us ? us + 0.1f * read_us : read_us + 0.1f * us);
    if (t < best) {
      best = t;
      *bn = w;
    }
  }
  return best;
}

// YAFSDP_GEMM_CTA_GROUP=1 in the environment: no CTA pairs where a single CTA can do the work
bool single_ctas_only() {
  static const bool single = [] {
    const char* v = getenv("YAFSDP_GEMM_CTA_GROUP");
    return v && atoi(v) == 1;
  }();
  return single;
}

// n_align > 0: tiles must end where multiples of n_align columns do (the pieces of B)
// kind: 0 bf16 output that may be computed swapped, 1 fp32 output, 2 any other
Plan make_plan(int M, int N, int K, int kind, int n_align, int sm_limit, bool may_split, int tile, int splits, float* us = nullptr) {
  const bool out_f32 = kind == 1;
  int sms = yf_num_sms();
  if (sm_limit > 0 && sm_limit < sms) sms = sm_limit;
  const int num_k = (K + BLOCK_K - 1) / BLOCK_K;
  Plan best = {0, 0, 1, 0, 0, 0};
  float best_c = 0.f;
  const bool single_ctas = single_ctas_only();
  for (int t = 1; t <= 5; ++t) {
    if ((tile > 0 && t != tile) || (tile == 0 && single_ctas && TILE_SHAPES[t].cg == 2)) continue;
    if (n_align > 0 && n_align % TILE_SHAPES[t].bn != 0) continue;
    const int units = sms / TILE_SHAPES[t].cg;
    if (units < 1) continue;
    for (int sp = 1; sp <= MAX_SPLITS; ++sp) {
      if (sp > 1 && (!may_split || num_k < 4 * sp)) break;
      if (splits > 0 && sp != splits && !(sp == 1 && num_k < 4 * splits)) continue;
      const float c = plan_us(TILE_SHAPES[t], M, N, K, units, sp, out_f32);
      if (best.tile == 0 || c < best_c) {
        best.tile = t;
        best.splits = sp;
        best_c = c;
      }
    }
  }
  if (kind == 0 && ((tile == 0 && !single_ctas) || tile == TILE_SWAP) && splits <= 1 && n_align % 256 == 0 && sms >= 2) {
    int bn = 0;
    const float c = swap_us(M, N, K, sms / 2, &bn);
    if (bn > 0 && (best.tile == 0 || c < best_c)) {
      best = {TILE_SWAP, 0, 1, bn, 0, 0};
      best_c = c;
    }
  }
  if (us != nullptr) *us = best_c;
  if (best.tile == 0 || best.tile == TILE_SWAP) return best;
  const TileShape& t = TILE_SHAPES[best.tile];
  const int tile_m = BLOCK_M * t.cg, units = sms / t.cg;
  const long long tiles = (long long)((M + tile_m - 1) / tile_m) * ((N + t.bn - 1) / t.bn);
  best.split_tiles = (int)(tiles % units);
  if (best.split_tiles == 0) best.splits = 1;
  if (best.splits > 1) {
    const long long ctas = (long long)best.split_tiles * t.cg;
    best.counters = (ctas * 8 + 255) / 256 * 256;
    best.bytes = best.counters + ctas * best.splits * BLOCK_M * t.bn * 4;
  }
  return best;
}

unsigned long long next_nonce() {  // 56 bits, never 0, another one in each of 2^56 launches of this process
  static std::atomic<unsigned long long> n{0};
  // modulo 2^56 multiplication by an odd number permutes: neighbours in time get words that differ in many places
  return ((n.fetch_add(1, std::memory_order_relaxed) + 1) * 0x9E3779B97F4A7C15ull) & ((1ull << 56) - 1);
}

template <int MODE>
int launch_tile(int tile, const Operands* ops, int n_ops, const GemmArgs& args, const FusedArgs& fa, int sm_limit, cudaStream_t s) {
  switch (tile) {
    case TILE_PAIR256: return launch_gemm<256, 2, MODE>(ops, n_ops, args, fa, sm_limit, s);
    case TILE_256: return launch_gemm<256, 1, MODE>(ops, n_ops, args, fa, sm_limit, s);
    case TILE_128: return launch_gemm<128, 1, MODE>(ops, n_ops, args, fa, sm_limit, s);
    case TILE_64: return launch_gemm<64, 1, MODE>(ops, n_ops, args, fa, sm_limit, s);
    default: return launch_gemm<128, 2, MODE>(ops, n_ops, args, fa, sm_limit, s);
  }
}

// n_ops > 1: the pieces of B (ops[i].N or ops[i].K rows each), every one with the same A
int launch_plain(const Operands* ops, int n_ops, GemmArgs args, const FusedArgs& fa, int sm_limit, void* workspace,
                 long long workspace_bytes, int tile, int splits, cudaStream_t s) {
  int n_align = 0;
  if (n_ops > 1) {
    args.n_parts = n_ops;
    int end = 0;
    for (int i = 0; i < n_ops; ++i) {
      if (i > 0 && !args.b_mn) n_align = std::gcd(n_align, end);
      end += args.b_mn ? ops[i].K : ops[i].N;
      args.parts[i] = end;
    }
    for (int i = n_ops - 1; i < MAX_GROUP; ++i) args.parts[i] = INT_MAX;  // searches stop at the last piece
  }
  const bool ws = workspace != nullptr && (reinterpret_cast<uintptr_t>(workspace) & 255) == 0;
  const int kind = args.out_f32 ? 1 : (args.a_mn || args.accumulate ? 2 : 0);
  Plan p = make_plan(args.M, args.N, args.K, kind, n_align, sm_limit, true, tile, splits);
  if (p.splits > 1 && (!ws || p.bytes > workspace_bytes)) p = make_plan(args.M, args.N, args.K, kind, n_align, sm_limit, false, tile, 1);
  if (p.tile == 0) return -1;
  args.splits = p.splits;
  if (p.tile == TILE_SWAP) {
    Operands swapped[MAX_GROUP];
    for (int i = 0; i < n_ops; ++i) swapped[i] = {ops[i].B, ops[i].A, ops[i].ldb, ops[i].lda, ops[i].N, ops[i].M, ops[i].K};
    std::swap(args.M, args.N);
    args.a_mn = args.b_mn;
    args.b_mn = 0;
    args.bn = p.bn;
    return launch_gemm<256, 2, MODE_SWAP>(swapped, n_ops, args, fa, sm_limit, s);
  }
  if (p.splits > 1) {
    args.split_tiles = p.split_tiles;
    args.nonce = next_nonce();
    args.counters = static_cast<unsigned long long*>(workspace);
    args.slots = reinterpret_cast<float*>(static_cast<uint8_t*>(workspace) + p.counters);
    return launch_tile<MODE_SPLIT>(p.tile, ops, n_ops, args, fa, sm_limit, s);
  }
  return launch_tile<MODE_PLAIN>(p.tile, ops, n_ops, args, fa, sm_limit, s);
}

// The entries without a workspace.  Plain mode: make_plan, nothing split.  Tile shape of the fused modes: CTA pairs (256 x 256 tiles,
// half of B per CTA) whenever both extents fill such a tile; single CTAs with 128 x 256 or 128 x 128 tiles for small or ragged
// problems.
int dispatch_gemm(const void* A, const void* B, const GemmArgs& args, const FusedArgs& fa, long long lda, long long ldb, int sm_limit,
                  cudaStream_t s) {
  const int M = args.M, N = args.N;
  const bool use256 = (N >= 256) && ((N % 256 == 0) || (N % 256 > 128) || N >= 2048);
  const bool single_ctas = single_ctas_only();
  const bool pair_ok = use256 && M >= 256 && (M % 256 == 0 || M % 256 > 128 || M >= 2048);
  if (fa.gather) {
    if (pair_ok && !single_ctas) return launch_gemm<256, 2, MODE_GATHER>(A, B, args, fa, lda, ldb, sm_limit, s);
    return use256 ? launch_gemm<256, 1, MODE_GATHER>(A, B, args, fa, lda, ldb, sm_limit, s)
                  : launch_gemm<128, 1, MODE_GATHER>(A, B, args, fa, lda, ldb, sm_limit, s);
  }
  if (fa.scatter) {
    if (pair_ok && !single_ctas) return launch_gemm<256, 2, MODE_SCATTER>(A, B, args, fa, lda, ldb, sm_limit, s);
    return use256 ? launch_gemm<256, 1, MODE_SCATTER>(A, B, args, fa, lda, ldb, sm_limit, s)
                  : launch_gemm<128, 1, MODE_SCATTER>(A, B, args, fa, lda, ldb, sm_limit, s);
  }
  const Operands one = {A, B, lda, ldb, M, N, args.K};
  return launch_plain(&one, 1, args, fa, sm_limit, nullptr, 0, single_ctas ? (use256 ? TILE_256 : TILE_128) : 0, 0, s);
}

}  // namespace

// C[M,N] = alpha * A * B^T (+ C).  A is [M,K] with row pitch lda (a_mn = 0) or stored as [K,M] with row
// pitch lda (a_mn = 1); B likewise as [N,K] (b_mn = 0) or [K,N] (b_mn = 1).  bf16 inputs; C is bf16 or
// fp32 (out_f32) with row pitch ldc.  Pitches are in elements and must be multiples of 8 (16-byte TMA
// strides); base pointers must be 16-byte aligned.  sm_limit > 0 caps the persistent grid (leaves SMs
// to a concurrent communication kernel).
extern "C" int yf_gemm_bf16_sumsq(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                                  long long ldc, int a_mn, int b_mn, int out_f32, int accumulate, float alpha, int sm_limit,
                                  float* sumsq, void* stream);

extern "C" int yf_gemm_bf16(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                            long long ldc, int a_mn, int b_mn, int out_f32, int accumulate, float alpha, int sm_limit,
                            void* stream) {
  return yf_gemm_bf16_sumsq(A, B, C, M, N, K, lda, ldb, ldc, a_mn, b_mn, out_f32, accumulate, alpha, sm_limit, nullptr, stream);
}

// Same as yf_gemm_bf16; when `sumsq` is given (fp32 output, no accumulation) the kernel also adds the sum of squares
// of everything it wrote to *sumsq, so a gradient norm needs no extra pass over a freshly written weight gradient.
extern "C" int yf_gemm_bf16_sumsq(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
                                  long long ldc, int a_mn, int b_mn, int out_f32, int accumulate, float alpha, int sm_limit,
                                  float* sumsq, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if (sumsq != nullptr && (!out_f32 || accumulate)) return -1;
  if ((lda % 8) || (ldb % 8) || (ldc % (out_f32 ? 4 : 8))) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = C;
  args.M = M; args.N = N; args.K = K;
  args.ldc = ldc;
  args.alpha = alpha;
  args.a_mn = a_mn ? 1 : 0;
  args.b_mn = b_mn ? 1 : 0;
  args.out_f32 = out_f32 ? 1 : 0;
  args.accumulate = accumulate ? 1 : 0;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  fa.sumsq = sumsq;
  return dispatch_gemm(A, B, args, fa, lda, ldb, sm_limit, s);
}

// C[M,N] = alpha * A * B^T + R with a bf16 residual R [M,N] (row pitch ldr) added in fp32 before the bf16 output is rounded;
// C may be R itself.  N, ldr multiples of 8; R 16-byte aligned.
extern "C" int yf_gemm_bf16_residual(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda,
                                     long long ldb, long long ldc, long long ldr, int a_mn, int b_mn, float alpha, int sm_limit,
                                     void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || R == nullptr) return -1;
  if ((lda % 8) || (ldb % 8) || (ldc % 8) || (ldr % 8) || (N % 8) || (reinterpret_cast<uintptr_t>(R) & 15)) return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = C;
  args.M = M; args.N = N; args.K = K;
  args.ldc = ldc;
  args.alpha = alpha;
  args.a_mn = a_mn ? 1 : 0;
  args.b_mn = b_mn ? 1 : 0;
  args.R = R;
  args.ldr = ldr;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  return dispatch_gemm(A, B, args, fa, lda, ldb, sm_limit, reinterpret_cast<cudaStream_t>(stream));
}

// The general form of the entries above.  `workspace` (256-byte aligned device memory that no other launch uses meanwhile, its
// contents do not matter) lets the last wave's tiles be split along K; yf_gemm_workspace says how much a problem wants, with
// less (or none) no tile is split.  kind: 0 bf16 output of a K-major A, 1 fp32 output, 2 any other.  tile,
// splits: 0 = chosen from the shape (make_plan); else a Tile (TILE_SWAP with kind 0 only) and 1 to MAX_SPLITS.
extern "C" int yf_gemm_workspace(int M, int N, int K, int kind, int n_align, int sm_limit, int tile, int splits, long long* bytes) {
  if (M <= 0 || N <= 0 || K <= 0 || kind < 0 || kind > 2 || n_align < 0 || bytes == nullptr || tile < 0 || tile > 6 || splits < 0 || splits > MAX_SPLITS) return -1;
  *bytes = make_plan(M, N, K, kind, n_align, sm_limit, true, tile, splits).bytes;
  return 0;
}
// the Tile that is chosen, plus 16 * (K ranges of the last wave's tiles); kind and n_align as above
extern "C" int yf_gemm_plan(int M, int N, int K, int kind, int n_align, int sm_limit) {
  if (M <= 0 || N <= 0 || K <= 0 || kind < 0 || kind > 2 || n_align < 0) return -1;
  const Plan p = make_plan(M, N, K, kind, n_align, sm_limit, true, 0, 0);
  return p.tile + 16 * p.splits;
}
extern "C" int yf_gemm_bf16_ws(const void* A, const void* B, void* C, const void* R, int M, int N, int K, long long lda, long long ldb,
                               long long ldc, long long ldr, int a_mn, int b_mn, int out_f32, int accumulate, float alpha, int sm_limit,
                               const float* alpha_ptr, float* sumsq, void* workspace, long long workspace_bytes, int tile, int splits, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || tile < 0 || tile > 6 || splits < 0 || splits > MAX_SPLITS) return -1;
  if (sumsq != nullptr && (!out_f32 || accumulate)) return -1;
  if ((lda % 8) || (ldb % 8) || (ldc % (out_f32 ? 4 : 8))) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return -1;
  if (R != nullptr && (out_f32 || accumulate || (ldr % 8) || (N % 8) || (reinterpret_cast<uintptr_t>(R) & 15))) return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = C;
  args.M = M; args.N = N; args.K = K;
  args.ldc = ldc;
  args.alpha = alpha;
  args.a_mn = a_mn ? 1 : 0;
  args.b_mn = b_mn ? 1 : 0;
  args.out_f32 = out_f32 ? 1 : 0;
  args.accumulate = accumulate ? 1 : 0;
  args.alpha_ptr = alpha_ptr;
  args.R = R;
  args.ldr = ldr;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  fa.sumsq = sumsq;
  const Operands one = {A, B, lda, ldb, M, N, K};
  return launch_plain(&one, 1, args, fa, sm_limit, workspace, workspace_bytes, tile, splits, reinterpret_cast<cudaStream_t>(stream));
}

// C[M,N] = A * B^T (bf16 output) with B in n (2 to 4) pieces of memory, one below the other: rows[i] rows of its storage ([N,K], or
// [K,N] with b_mn) at B[i], row pitch ldb[i].  Several weights of one layer act as one matrix without being copied together.
// Every piece but the last has a multiple of 64 rows.  n_align of yf_gemm_workspace: the greatest common divisor of the
// places where a piece of [N,K] storage starts; 0 with b_mn.
extern "C" int yf_gemm_bf16_parts(const void* A, int n, const void* const* B, const int* rows, const long long* ldb, void* C, int M,
                                  int N, int K, long long lda, long long ldc, int b_mn, void* workspace, long long workspace_bytes,
                                  int tile, int splits, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || n < 2 || n > MAX_GROUP || tile < 0 || tile > 6 || splits < 0 || splits > MAX_SPLITS) return -1;
  if ((lda % 8) || (ldc % 8) || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(C)) & 15)) return -1;
  Operands ops[MAX_GROUP];
  long long total = 0;
  for (int i = 0; i < n; ++i) {
    if (rows[i] <= 0 || (i + 1 < n && rows[i] % 64) || (ldb[i] % 8) || (reinterpret_cast<uintptr_t>(B[i]) & 15)) return -1;
    total += rows[i];
    ops[i] = {A, B[i], lda, ldb[i], M, b_mn ? N : rows[i], b_mn ? rows[i] : K};
  }
  if (total != (b_mn ? K : N)) return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = C;
  args.M = M; args.N = N; args.K = K;
  args.ldc = ldc;
  args.alpha = 1.f;
  args.b_mn = b_mn ? 1 : 0;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  return launch_plain(ops, n, args, fa, 0, workspace, workspace_bytes, tile, splits, reinterpret_cast<cudaStream_t>(stream));
}

// act[M,F] = silu(X Wg^T) * (X Wu^T) with Wg, Wu [F,K] (row pitches ldg, ldu); gu [M,2F] (may be null: not wanted) receives both
// products.  F a multiple of 128.
extern "C" int yf_gemm_swiglu(const void* X, const void* Wg, const void* Wu, void* gu, void* act, int M, int F, int K, long long ldx,
                              long long ldg, long long ldu, long long ldgu, long long ldact, void* stream) {
  if (M <= 0 || F <= 0 || K <= 0 || (F % 128) || (ldx % 8) || (ldg % 8) || (ldu % 8) || (ldact % 8) || (gu && (ldgu % 8))) return -1;
  if ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(Wg) | reinterpret_cast<uintptr_t>(Wu) | reinterpret_cast<uintptr_t>(gu) |
       reinterpret_cast<uintptr_t>(act)) & 15)
    return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = gu ? gu : act;  // without gu only a store map that nothing uses
  args.M = M; args.N = 2 * F; args.K = K;
  args.ldc = gu ? ldgu : ldact;
  args.alpha = 1.f;
  args.R = act;
  args.ldr = ldact;
  args.store_gu = gu != nullptr;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  const Operands ops[2] = {{X, Wg, ldx, ldg, M, F, K}, {X, Wu, ldx, ldu, M, F, K}};
  return launch_gemm<256, 2, MODE_SWIGLU>(ops, 2, args, fa, 0, reinterpret_cast<cudaStream_t>(stream));
}
// Whether that is estimated to be faster than the best plain GEMM and a separate activation kernel (6 bytes per element of act
// at 4 TB/s, 3 us).  The epilogue of a tile takes 11.3 us (exponentials, divisions and three stores in four warps), 2.7 us of it also a
// plain tile's; the next tile's main loop hides it, but not the last one's, and where K is short it hides the main loop.  Measured in
// a stream of launches at the power cap, GEMM + activation / fused, us:
//   F 11008, K 4096: 45 tokens 47 / 62, 300 72 / 84, 777 145 / 157, 999 175 / 158, 1337 222 / 216, 2048 323 / 284, 8192 1201 / 1015
//   F 14336, K 4096: 777 tokens 176 / 199, 1337 282 / 291, 2048 421 / 365;  F 13824, K 5120: 300 tokens 98 / 116, 512 137 / 133
//   F 28672, K 8192: 128 tokens 177 / 215, 777 686 / 757, 1337 1084 / 1098, 2048 1696 / 1534, 4096 3249 / 2957
// (While rows past the end went through the epilogue's divisions, which take several times as long for 0 / x, fused tiles with such
// rows cost 12 us more each: 1337 tokens 240, 777 187, 300 126 us at F 11008.)
extern "C" int yf_gemm_swiglu_pays(int M, int F, int K) {
  if (M <= 0 || F <= 0 || K <= 0) return -1;
  if ((F % 128) || single_ctas_only()) return 0;  // the fused kernel has CTA pairs only
  const int sms = yf_num_sms(), num_k = (K + BLOCK_K - 1) / BLOCK_K;
  float best = 0.f;
  make_plan(M, 2 * F, K, 0, 0, 0, true, 0, 0, &best);
  const TileShape& t = TILE_SHAPES[TILE_PAIR256];
  const long long tiles = (long long)((M + 255) / 256) * (F / 128), units = sms / 2;
  const float loop = (float)num_k * t.kb_us, epi = 11.3f, longer = loop > epi ? loop : epi, shorter = loop > epi ? epi : loop;
  const float us = (float)((tiles + units - 1) / units) * longer, read_us = ((float)M + 2.f * (float)F) * (float)K * 2.f / 5.2e6f;
  const float fused = t.fixed_us + shorter - 2.7f + (us > read_us ? us + 0.1f * read_us : read_us + 0.1f * us);  // as in plan_us
  return fused <= best + 3.f + (float)M * (float)F * 6.f / 4e6f ? 1 : 0;
}

// All-gather -> GEMM in one kernel.  C[M,N] = A[M,K] * B[N,K]^T where B (row-major, contiguous, K-major) is a
// sub-range of the layer's flat bf16 parameter buffer that the same kernel gathers:
//   peer_in[r]  : rank r's shard (shard_bytes bytes) of the layer, peer-mapped; entry `rank` is the local shard
//   layer_buf   : local unsharded layer buffer (world * shard_bytes bytes); B = layer_buf + b_byte_off
//   counters    : one unsigned 64-bit word per B column block of 256 rows (128 when N < 256), in this GPU's memory, zero
//                 before the first call; epoch = 1, 2, ... counts the calls made with these counters and this shape
// On return (stream order) the whole layer buffer is filled, not only B.
extern "C" int yf_gemm_bf16_gathered(const void* A, void* C, int M, int N, int K, long long lda, long long ldc, int a_mn,
                                     int out_f32, void* const* peer_in, void* layer_buf, long long shard_bytes,
                                     long long b_byte_off, int rank, int world, void* counters, long long epoch, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || world < 1 || world > MAX_RANKS || rank < 0 || rank >= world) return -1;
  if ((lda % 8) || (K % 8) || (ldc % (out_f32 ? 4 : 8)) || epoch <= 0 || counters == nullptr) return -1;
  if ((shard_bytes % 16) || shard_bytes <= 0 || (b_byte_off % 16)) return -1;
  if (b_byte_off < 0 || b_byte_off + (long long)N * K * 2 > shard_bytes * world) return -1;
  const uint8_t* B = reinterpret_cast<const uint8_t*>(layer_buf) + b_byte_off;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
       reinterpret_cast<uintptr_t>(layer_buf)) & 15)
    return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = C;
  args.M = M; args.N = N; args.K = K;
  args.ldc = ldc;
  args.alpha = 1.f;
  args.a_mn = a_mn ? 1 : 0;
  args.b_mn = 0;
  args.out_f32 = out_f32 ? 1 : 0;
  args.accumulate = 0;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  fa.gather = 1;
  fa.world = world; fa.rank = rank;
  fa.counters = reinterpret_cast<unsigned long long*>(counters);
  fa.epoch = (unsigned long long)epoch;
  for (int r = 0; r < world; ++r) {
    if (!peer_in[r] || (reinterpret_cast<uintptr_t>(peer_in[r]) & 15)) return -1;
    fa.peer_in[r] = peer_in[r];
  }
  fa.layer_buf = reinterpret_cast<uint8_t*>(layer_buf);
  fa.shard_bytes = shard_bytes;
  fa.b_byte_off = b_byte_off;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return dispatch_gemm(A, B, args, fa, lda, K, 0, s);
}

// GEMM -> reduce-scatter in one kernel.  dW[M,N] = A * B^T in fp32 is not stored locally: each 16-byte piece is
// pushed into the staging slot `rank` of the rank that owns its position c_flat_off + m*N + n of the flat layer
// gradient (peer_grad[o] = base of owner o's reduce buffer, laid out as `world` slots of shard_numel floats).
// wire_bf16: the slots hold bf16 instead of fp32 (half the NVLink bytes; the owner still sums in fp32).  shard_numel, N and
// c_flat_off must be multiples of 4 (8 with the bf16 wire).  The owners sum their slots afterwards
// (yf_reduce_scatter_pull on local slot pointers) once every rank's pushes are complete.
extern "C" int yf_gemm_bf16_scatter(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int a_mn,
                                    int b_mn, float alpha, void* const* peer_grad, long long c_flat_off, long long shard_numel,
                                    int rank, int world, int wire_bf16, int sm_limit, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0 || world < 1 || world > MAX_RANKS || rank < 0 || rank >= world) return -1;
  const int al = wire_bf16 ? 8 : 4;  // elements per 16 bytes on the wire
  if ((lda % 8) || (ldb % 8) || (N % al) || (shard_numel % al) || (c_flat_off % al) || c_flat_off < 0) return -1;
  if (c_flat_off + (long long)M * N > shard_numel * world) return -1;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  args.C = peer_grad[rank];  // only used to build a (unused) store descriptor
  args.M = M; args.N = N; args.K = K;
  args.ldc = N;
  args.alpha = alpha;
  args.a_mn = a_mn ? 1 : 0;
  args.b_mn = b_mn ? 1 : 0;
  args.out_f32 = 1;
  args.accumulate = 0;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  fa.scatter = 1;
  fa.wire_bf16 = wire_bf16 ? 1 : 0;
  fa.world = world; fa.rank = rank;
  for (int r = 0; r < world; ++r) {
    if (!peer_grad[r] || (reinterpret_cast<uintptr_t>(peer_grad[r]) & 15)) return -1;
    fa.peer_grad[r] = peer_grad[r];
  }
  fa.c_flat_off = c_flat_off;
  fa.shard_numel = shard_numel;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return dispatch_gemm(A, B, args, fa, lda, ldb, sm_limit, s);
}

// The weight-gradient GEMMs of a whole layer as ONE launch, pushed to their owners (grouped GEMM -> reduce-scatter).
// n problems (at most 4) dW_i[M_i, N_i] = A_i^T-or-not * B_i, sharing K and the operand majors, in the order of their
// positions flat_off[i] in the flat layer gradient.  Every rank deals the owners' tiles round-robin (owner rank + 1 first), so
// it pushes to all owners all the time and no owner's NVLink ingress becomes a hot spot, which separate launches cannot
// avoid (all ranks would push the same rows, i.e. to the same one or two owners, at the same time).
extern "C" int yf_gemm_bf16_scatter_grouped(int n, const void* const* A, const void* const* B, const int* M, const int* N, int K,
                                            const long long* lda, const long long* ldb, int a_mn, int b_mn, float alpha,
                                            void* const* peer_grad, const long long* flat_off, long long shard_numel, int rank,
                                            int world, int wire_bf16, int sm_limit, void* stream) {
  const int al = wire_bf16 ? 8 : 4;  // elements per 16 bytes on the wire
  if (n < 1 || n > MAX_GROUP || K <= 0 || world < 1 || world > MAX_RANKS || rank < 0 || rank >= world || (shard_numel % al)) return -1;
  GemmArgs args;
  memset(&args, 0, sizeof(args));
  Operands ops[MAX_GROUP];
  bool all256 = true;
  for (int i = 0; i < n; ++i) {
    if (M[i] <= 0 || N[i] <= 0 || (lda[i] % 8) || (ldb[i] % 8) || (N[i] % al) || (flat_off[i] % al) || flat_off[i] < 0) return -1;
    if (flat_off[i] + (long long)M[i] * N[i] > shard_numel * world) return -1;
    if (i > 0 && flat_off[i] < flat_off[i - 1] + (long long)M[i - 1] * N[i - 1]) return -1;  // ascending, no overlap
    if ((reinterpret_cast<uintptr_t>(A[i]) | reinterpret_cast<uintptr_t>(B[i])) & 15) return -1;
    ops[i] = {A[i], B[i], lda[i], ldb[i], M[i], N[i], K};
    args.Mp[i] = M[i];
    args.Np[i] = N[i];
    args.flat_off[i] = flat_off[i];
    all256 = all256 && M[i] >= 256 && N[i] >= 256;
  }
  args.n_prob = n;
  args.C = peer_grad[rank];  // only used to build a (unused) store descriptor
  args.M = M[0]; args.N = N[0]; args.K = K;
  args.ldc = N[0];
  args.alpha = alpha;
  args.a_mn = a_mn ? 1 : 0;
  args.b_mn = b_mn ? 1 : 0;
  args.out_f32 = 1;
  FusedArgs fa;
  memset(&fa, 0, sizeof(fa));
  fa.scatter = 1;
  fa.wire_bf16 = wire_bf16 ? 1 : 0;
  fa.world = world; fa.rank = rank;
  for (int r = 0; r < world; ++r) {
    if (!peer_grad[r] || (reinterpret_cast<uintptr_t>(peer_grad[r]) & 15)) return -1;
    fa.peer_grad[r] = peer_grad[r];
  }
  fa.shard_numel = shard_numel;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (all256) return launch_gemm<256, 2, MODE_SCATTER>(ops, n, args, fa, sm_limit, s);
  return launch_gemm<128, 1, MODE_SCATTER>(ops, n, args, fa, sm_limit, s);
}
