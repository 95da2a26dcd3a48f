// Row-parallel GEMM with an NVFP4 epilogue that pushes straight into the AllReduce receive windows.
//
//   partial[M, N] = X[M, K] (BF16, K contiguous) x Wt[N, K]^T (BF16, K contiguous), FP32 accumulate
//   epilogue: every 16 consecutive outputs of a row are quantised with the static per-rank scale gs
//             (block scale e4m3(rn(rn(blockmax/gs')/6)), values e2m1, -0 canonicalised: the static-scale row
//             format of the AllReduce), and the row pieces are stored
//               - into every rank's receive window (one-shot), or into the row owner's window (two-shot),
//                 where the AllReduce kernel in "pushed input" mode finds them, and/or
//               - into a local [M, N/2 + N/16] NVFP4 tensor.
//
// sm_100a structure: up to 384 rows one narrow tile per CTA (gemm_narrow_kernel below); above that persistent CTAs (one
// per SM), K in blocks of 64, three shapes:
//   pairs  (default for K >= 4096 or M >= 8192): the two CTAs of a cluster share one 256 x 256 tile with tcgen05
//          cta_group::2: each loads its own 128 rows of A and half of the B block into a 6-stage ring, the even CTA
//          issues the MMAs for both, each CTA's TMEM holds the accumulator of its own 128 rows;
//   single: one CTA per 128 x 256 tile (4-stage ring) or 128 x 192 tile (5-stage ring, where that fills the last wave
//          of CTAs better and the K split below does not apply).
// Where the tile count is not a multiple of the unit count (CTAs or pairs), the first (units + remainder) tiles are cut
// along K into equal ranges per unit (stream-K, see SegIter) so that no SM idles through a last wave.
//   warp 0  : TMA producer   - cp.async.bulk.tensor (every CTA loads for itself) of the A and B blocks into the ring,
//                              128-byte swizzle, completion on mbarriers (of a pair: both CTAs' bytes are counted
//                              under the leader's barrier)
//   warp 1  : MMA issuer     - one thread issues tcgen05.mma (kind::f16, M 128 per CTA, N 256, K 16) from
//                              shared-memory descriptors into TMEM; tcgen05.commit releases ring stages and
//                              publishes finished accumulators (of a pair: on both CTAs' barriers); owns
//                              tcgen05.alloc / dealloc (512 columns = two accumulators, so the epilogue of tile i
//                              overlaps the main loop of tile i+1)
//   warps 2-5: epilogue      - tcgen05.ld (32 lanes x 32 columns per instruction), quantise, stage the row
//                              pieces in shared memory, bulk-store them to the (peer) windows
// Every wait is bounded; a wait that gives up raises a CTA-wide abort flag, the roles drain, TMEM is freed and
// the status word reports it.
//
// The reference project has no such producer: its NVFP4-input kernels assume one and the harness emulates it
// with a copy (README.md:76, docs/INTEGRATION.md:67-74, harness/fp4ar_bench.cu:205-215).
#include <cuda.h>
#include <cuda_runtime.h>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <optional>
#include <vector>
#include "../include/fp4ar.h"
#include "../include/fp4ar_codec.cuh"
#include "../include/fp4ar_async.cuh"
#include "../include/fp4ar_gemm.h"
#include "host_util.h"

namespace fp4ar {

constexpr int kBM = 128, kBK = 64;
constexpr int kABytes = kBM * kBK * 2;            // 16 KB
constexpr int kGemmThreads = 192;
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxStages = 6;

// Tile width BN: 256 with a 4-stage ring, or 192 with a 5-stage ring.  With 148 persistent CTAs the tile count decides
// how full the last wave is: M = 1024, N = 6144 gives 192 tiles of 128 x 256 (1.3 waves, 65 % busy) but 256 tiles of
// 128 x 192 (1.7 waves, 86 % busy).  (A 128-wide tile with a 6-stage ring was measured 15-35 % slower at every M from
// 1024 to 4096 and is not built.)
// G = 2: two CTAs of a cluster (an SM pair) work on one 256 x 256 tile with tcgen05 cta_group::2: each CTA loads its own
// 128 rows of A and HALF of the B block (128 of the 256 columns), the tensor cores of both SMs read both halves, and
// each CTA's TMEM holds the accumulator of its own 128 rows.  A K block then costs a CTA 32 KB of shared-memory fill
// instead of 48 KB, and the ring is six stages deep.
template <int BN, int G = 1>
struct GemmShape {
  static_assert(BN == 256 || BN == 192, "tile width");
  static_assert(G == 1 || (G == 2 && BN == 256), "CTA pairs use the 256-wide tile");
  static constexpr int kStages = G == 2 ? 6 : (BN == 256 ? 4 : 5);
  static constexpr int kBBytes = BN / G * kBK * 2;              // 32 KB / 24 KB, 16 KB per CTA of a pair
  static constexpr int kStageBytes = kABytes + kBBytes;         // 48 KB / 40 KB / 32 KB
  static constexpr int kTxBytes = kStageBytes * G;              // what lands per stage under the (leader's) full barrier
  static constexpr int kValueB = BN / 2, kScaleB = BN / 16;     // 128 + 16 B / 96 + 12 B of one row of one tile
  static constexpr int kPieceBytes = (kValueB + kScaleB + 15) & ~15;   // 144 / 112: keeps every piece 16-byte aligned
  static constexpr int kEpiBytes = kBM * kPieceBytes;
  static constexpr int kSmem = kStages * kStageBytes + kEpiBytes + 256 + 1024;   // + barriers + alignment slack
  // Instruction descriptor: D = F32, A = B = BF16, both K-major, N = BN, M = 128 per CTA of the group.
  static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((kBM * G) >> 4) << 24);
};

struct GemmParams {
  int M, N, K;
  float inv_gs;
  // push destination (nranks == 0: none)
  char* win[kMaxRanksOps];
  const uint32_t* call_counter;
  unsigned long long buf_bytes;
  int cap, capo, nranks, rank, two_shot;
  // local outputs (optional)
  char* local_q;       // [M][N/2 + N/16]
  float* dbg_acc;      // [M][N]
  StatusWords* status;
  unsigned long long timeout_ns;
  // split of the K loop across CTAs (see SegIter): partial accumulators and their flags, one slot per CTA
  int a_rows, stages, atoms;    // few rows: rows of the A box, ring stages, K blocks per stage (see gemm_narrow_kernel)
  int stream_k;
  float* sk_partial;     // [grid][BN / 32][8][128] float4
  uint32_t* sk_flags;    // [grid][4]: 1 = the slot's quarter (32 rows) is written and not yet consumed
};

// ---- tcgen05 / TMA wrappers ----
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_addr(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar))
               : "memory");
}
// `z` counts K blocks: a box of several lands as consecutive [rows][128 bytes] tiles
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int y, int z, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(smem_addr(smem_dst)), "l"(map), "r"(0), "r"(y), "r"(z), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void prefetch_tensormap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* holder, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(holder)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{ .reg .pred p;\n"
               "  setp.ne.b32 p, %4, 0;\n"
               "  tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p; }"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
               : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// ---- CTA pair (cluster of two) ----
__device__ __forceinline__ uint32_t cluster_cta_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of the same shared-memory location in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(const void* local, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(local)), "r"(rank));
  return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
// TMA load of one CTA of a pair: the bytes are counted under the barrier at `cluster_bar` (the leader's); every CTA loads for itself
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t cluster_bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
               ::"r"(smem_addr(smem_dst)), "l"(map), "r"(x), "r"(y), "r"(cluster_bar)
               : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* holder, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(holder)), "r"(cols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() { asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t addr, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(cols) : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile("{ .reg .pred p;\n"
               "  setp.ne.b32 p, %4, 0;\n"
               "  tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p; }"
               ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
               : "memory");
}
// arrives on the barrier at the same shared-memory offset in both CTAs of the pair once the MMAs issued so far are done
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("{ .reg .b16 m;\n"
               "  mov.b16 m, 3;\n"
               "  tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m; }"
               ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// Starts the load of 32 accumulator columns of this thread's TMEM lane; the registers are valid after tmem_ld_wait().
__device__ __forceinline__ void tmem_ld32_issue(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
               "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
               "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                 "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                 "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
               : "r"(taddr));
}
// All tcgen05.ld of this thread issued so far have delivered their registers.
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile whose rows are 128 bytes (64 BF16) with the 128-byte
// swizzle: 8-row groups 1024 bytes apart, descriptor version 1 (sm_100), layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_k128(const void* smem_tile) {
  uint64_t d = (uint64_t)((smem_addr(smem_tile) >> 4) & 0x3FFFu);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused with a swizzle), in 16-byte units
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;            // version
  d |= (uint64_t)2 << 61;            // SWIZZLE_128B
  return d;
}

// Tile order: the N tiles are walked in panels of kPanel; inside a panel consecutive tile indices step through
// N fastest and then M.  The ~148 tiles in flight at a time then cover about 18 row blocks x 8 column tiles, which
// needs (18 + 2*8) * 128 * K * 2 bytes of operands from L2 instead of (6 + 2*24) for a plain row-major walk.
constexpr int kPanel = 8;
template <int BN, int G = 1>
__device__ __forceinline__ void tile_coords(int t, int m_tiles, int n_tiles, int& m0, int& n0) {
  const int per_panel = m_tiles * kPanel;
  const int panel = t / per_panel, within = t - panel * per_panel;
  const int width = min(kPanel, n_tiles - panel * kPanel);
  const int m = within / width, n = panel * kPanel + within % width;
  m0 = m * kBM * G; n0 = n * BN;
}

struct GemmWait {
  volatile uint32_t* abort_flag;
  StatusWords* status;
  unsigned long long limit_ns;
};
// Bounded mbarrier wait; false when it gave up or the CTA is aborting.
__device__ __forceinline__ bool gemm_wait(uint64_t* bar, uint32_t parity, const GemmWait& w, uint32_t what) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = global_timer_ns();
  uint32_t n = 0;
  while (!mbar_test(bar, parity)) {
    if ((++n & 255u) == 0u) {
      if (*w.abort_flag) return false;
      if (global_timer_ns() - t0 > w.limit_ns) {
        *w.abort_flag = 1u;
        if (atomicCAS(&w.status->code, 0u, (uint32_t)kStatusLoadTimeout) == 0u) { w.status->detail = 16u + what; w.status->cta = blockIdx.x; }
        atomicAdd(&w.status->count, 1u);
        return false;
      }
    }
  }
  return true;
}

// A CTA that gives up may still have copies on their way into its shared memory and MMAs at work on its TMEM: it leaves only
// when their barrier says that they are through (10 ms at most).
__device__ __forceinline__ void gemm_settle(uint64_t* bar, uint32_t parity) {
  const unsigned long long t0 = global_timer_ns();
  while (!mbar_test(bar, parity) && global_timer_ns() - t0 < 10000000ull) {}
}

// Bounded wait until *flag == want (acquire); false when it gave up or the CTA is aborting.
__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ bool gemm_flag_wait(const uint32_t* flag, uint32_t want, const GemmWait& w, uint32_t what) {
  if (ld_acquire_gpu(flag) == want) return true;
  const unsigned long long t0 = global_timer_ns();
  uint32_t n = 0;
  while (ld_acquire_gpu(flag) != want) {
    if ((++n & 63u) == 0u) {
      if (*w.abort_flag) return false;
      if (global_timer_ns() - t0 > w.limit_ns) {
        *w.abort_flag = 1u;
        if (atomicCAS(&w.status->code, 0u, (uint32_t)kStatusLoadTimeout) == 0u) { w.status->detail = 16u + what; w.status->cta = blockIdx.x; }
        atomicAdd(&w.status->count, 1u);
        return false;
      }
    }
  }
  return true;
}

// The work of one CTA as a list of segments (tile, K blocks [lo, lo + count), rotation), the same list in all three roles.
//   plain:    whole tiles blockIdx.x, blockIdx.x + grid, ...
//   stream-K: with tiles = w * grid + r (0 < r < grid) the first grid + r tiles are cut, as tiles x kblocks units,
//             into `grid` equal contiguous ranges, so every CTA runs the same number of K blocks there (between one and
//             two tiles' worth) instead of r CTAs running one more tile than the others; the other (w - 1) * grid
//             tiles follow as whole tiles.  A range is at least one tile long, so a tile is shared by at most two
//             CTAs: the one whose range BEGINS inside the tile (kProduce) runs its share first, on the tile's FIRST K
//             blocks, and leaves its FP32 accumulator in its slot of the partial buffer; the one whose range ENDS
//             inside the tile (kFix) runs the remaining K blocks last, adds that partial and does the tile's epilogue.
//             The partial was written about one tile duration or more before it is read.
//   K order:  every segment walks its K blocks upwards.  The producing share is the tile's FIRST K blocks and the fixing
//             share its LAST ones, so a CTA that starts with a share of c blocks is at block t while it produces, at
//             t - c in the whole tile that follows and at most (range - kblocks) behind t in its fixing share: at
//             any moment all CTAs read 64-column slices of X and Wt that lie within that window of each other and no
//             slice is needed again after the window has passed, so the operands cross HBM once.  (Shares that start
//             at unrelated K offsets: 123 us at M = 1024, K = 8192; a cyclic walk locked to a common clock: 94 us,
//             267 MB of DRAM reads for 116 MB of operands because the wrapped part is re-read.)
enum : int { kWhole = 0, kProduce = 1, kFix = 2 };
struct Seg { int tile, lo, count, kind; };      // K blocks lo .. lo + count - 1
struct SegIter {
  int tiles, kblocks, stride, t;
  long long u, u_end;
  // unit = this CTA (or CTA pair) among `units` of them
  __host__ __device__ SegIter(int stream_k, int tiles_, int kblocks_, int unit, int units) : tiles(tiles_), kblocks(kblocks_), stride(units) {
    const int g = units;
    const int cut_tiles = stream_k ? g + tiles_ % g : 0;
    const long long total = (long long)cut_tiles * kblocks_;
    u = total * unit / g;
    u_end = total * (unit + 1) / g;
    t = cut_tiles + unit;
  }
  __host__ __device__ bool next(Seg& s) {
    if (u < u_end) {
      s.tile = (int)(u / kblocks);
      const int off = (int)(u - (long long)s.tile * kblocks);
      const long long left = u_end - u;
      const int room = kblocks - off;
      s.count = (int)(left < room ? left : room);
      if (off > 0) { s.kind = kProduce; s.lo = 0; }
      else if (s.count < kblocks) { s.kind = kFix; s.lo = kblocks - s.count; }
      else { s.kind = kWhole; s.lo = 0; }
      u += s.count;
    } else {
      if (t >= tiles) return false;
      s.tile = t; s.lo = 0; s.count = kblocks; s.kind = kWhole;
      t += stride;
    }
    return true;
  }
};

template <int BN, int G>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_nvfp4_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  const __grid_constant__ GemmParams p) {
  using S = GemmShape<BN, G>;
  constexpr int kStages = S::kStages, kStageBytes = S::kStageBytes, kEpiBytes = S::kEpiBytes, kPieceBytes = S::kPieceBytes;
  constexpr uint32_t kIdesc = S::kIdesc;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* ring = smem;
  uint8_t* epi = smem + kStages * kStageBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(epi + kEpiBytes);   // [kMaxStages]
  uint64_t* empty = full + kMaxStages;                              // [kMaxStages]
  uint64_t* acc_full = empty + kMaxStages;                          // [2]
  uint64_t* acc_empty = acc_full + 2;                               // [2]
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
  volatile uint32_t* abort_flag = tmem_holder + 1;
  uint64_t* settled = reinterpret_cast<uint64_t*>(tmem_holder + 2);
  uint32_t issued = 0;                 // ring stages that this CTA's producer has filled

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_tiles = p.N / BN, m_tiles = (p.M + kBM * G - 1) / (kBM * G);
  const int tiles = n_tiles * m_tiles, kblocks = p.K / kBK;
  // a pair works as one unit: the even CTA (cluster rank 0) leads, i.e. owns the barriers the MMAs wait on and issues them
  const uint32_t crank = G == 2 ? cluster_cta_rank() : 0u;
  const bool leads = crank == 0u;
  const int unit = blockIdx.x / G, units = gridDim.x / G;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; s++) { mbar_init(full + s, 1); mbar_init(empty + s, 1); }
    for (int a = 0; a < 2; a++) { mbar_init(acc_full + a, 1); mbar_init(acc_empty + a, 128 * G); }
    mbar_init(settled, 1);
    *abort_flag = 0u;
    mbar_init_fence();
  }
  if (warp == 1) {
    if constexpr (G == 2) { tmem_alloc_pair(tmem_holder, kTmemCols); tmem_relinquish_pair(); }
    else { tmem_alloc(tmem_holder, kTmemCols); tmem_relinquish(); }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (G == 2) cluster_sync_all();     // the partner's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  GemmWait gw{abort_flag, p.status, p.timeout_ns};

  pdl_wait_prior_grids();   // the windows and the call counter belong to the previous kernel until here
  pdl_release_dependents();

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      SegIter seg(p.stream_k, tiles, kblocks, unit, units);
      Seg sg;
      while (seg.next(sg)) {
        int m0, n0;
        tile_coords<BN, G>(sg.tile, m_tiles, n_tiles, m0, n0);
        for (int j = 0; j < sg.count; j++, issued++) {
          const int kb = sg.lo + j;
          const int s = issued % kStages;
          if (!gemm_wait(empty + s, ((issued / kStages) & 1u) ^ 1u, gw, 1)) goto done;
          if constexpr (G == 2) {
            // both CTAs' bytes are counted under the leader's barrier; only the leader announces them
            const uint32_t lead_full = cluster_addr(full + s, 0u);
            if (leads) mbar_arrive_expect(full + s, S::kTxBytes);
            tma_load_2d_pair(ring + s * kStageBytes, &map_a, kb * kBK, m0 + (int)crank * kBM, lead_full);
            tma_load_2d_pair(ring + s * kStageBytes + kABytes, &map_b, kb * kBK, n0 + (int)crank * (BN / 2), lead_full);
          } else {
            mbar_arrive_expect(full + s, kStageBytes);
            tma_load_2d(ring + s * kStageBytes, &map_a, kb * kBK, m0, full + s);
            tma_load_2d(ring + s * kStageBytes + kABytes, &map_b, kb * kBK, n0, full + s);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (of a pair: the leader's)
    if (lane == 0 && leads) {
      uint32_t it = 0, tile_i = 0;
      SegIter seg(p.stream_k, tiles, kblocks, unit, units);
      Seg sg;
      for (; seg.next(sg); tile_i++) {
        const uint32_t a = tile_i & 1u;
        if (!gemm_wait(acc_empty + a, ((tile_i >> 1) & 1u) ^ 1u, gw, 2)) goto done;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + a * BN;
        for (int j = 0; j < sg.count; j++, it++) {
          const int s = it % kStages;
          if (!gemm_wait(full + s, (it / kStages) & 1u, gw, 3)) goto done;
          tc_fence_after();
          const uint64_t da = umma_desc_k128(ring + s * kStageBytes);
          const uint64_t db = umma_desc_k128(ring + s * kStageBytes + kABytes);
#pragma unroll
          for (int k = 0; k < kBK / 16; k++) {
            if constexpr (G == 2) umma_bf16_pair(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), kIdesc, (j | k) != 0 ? 1u : 0u);
            else umma_bf16(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), kIdesc, (j | k) != 0 ? 1u : 0u);
          }
          // the stage is free once these MMAs have read it (of a pair: in both CTAs)
          if constexpr (G == 2) umma_commit_pair(empty + s); else umma_commit(empty + s);
        }
        // the accumulator is complete once everything above has run
        if constexpr (G == 2) umma_commit_pair(acc_full + a); else umma_commit(acc_full + a);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (warps 2..5 = 128 threads = 128 rows)
    const int q = warp & 3;                       // TMEM lane quarter this warp may read
    const int r_in_tile = q * 32 + lane;
    uint8_t* my_piece = epi + r_in_tile * kPieceBytes;
    const size_t buf_off = p.nranks ? (size_t)(*p.call_counter & 1u) * p.buf_bytes : 0;
    const int qrow_bytes = p.N / 2 + p.N / 16;
    uint32_t tile_i = 0;
    SegIter seg(p.stream_k, tiles, kblocks, unit, units);
    Seg sg;
    // this thread's float4 i of chunk c inside a partial slot: a warp's 32 rows are 512 contiguous bytes
    auto slot_ptr = [&](int cta, int c, int i) {
      return reinterpret_cast<float4*>(p.sk_partial) + ((size_t)cta * (BN / 32) + c) * 8 * kBM + (size_t)i * kBM + r_in_tile;
    };
    // 128 arrivals per CTA hand the accumulator back to the MMA warp (of a pair: to the leader's)
    auto hand_back = [&](uint32_t a) {
      if constexpr (G == 2) mbar_arrive_cluster(cluster_addr(acc_empty + a, 0u)); else mbar_arrive(acc_empty + a);
    };
    for (; seg.next(sg); tile_i++) {
      int m0, n0;
      tile_coords<BN, G>(sg.tile, m_tiles, n_tiles, m0, n0);
      m0 += (int)crank * kBM;                              // of a pair: this CTA's half of the 256 rows
      const uint32_t a = tile_i & 1u;
      const int row = m0 + r_in_tile;
      const bool produces = sg.kind == kProduce;           // a share of the tile's K blocks: leave a partial
      const bool fixes = sg.kind == kFix;                  // the rest of them: add the next CTA's partial
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16) + a * BN;
      if (produces) {
        // the slot is free once the consumer of an earlier launch has reset the flag
        uint32_t* flag = p.sk_flags + blockIdx.x * 4 + q;
        bool ok = lane == 0 ? gemm_flag_wait(flag, 0u, gw, 5) : true;
        ok = __all_sync(0xffffffffu, ok) && __all_sync(0xffffffffu, gemm_wait(acc_full + a, (tile_i >> 1) & 1u, gw, 4));
        if (!ok) break;
        tc_fence_after();
        float v[2][32];
        tmem_ld32_issue(tbase, v[0]);
#pragma unroll
        for (int c = 0; c < BN / 32; c++) {
          tmem_ld_wait();
          if (c + 1 < BN / 32) tmem_ld32_issue(tbase + (c + 1) * 32, v[(c + 1) & 1]);
          const float* vc = v[c & 1];
#pragma unroll
          for (int i = 0; i < 8; i++) *slot_ptr(blockIdx.x, c, i) = make_float4(vc[4 * i], vc[4 * i + 1], vc[4 * i + 2], vc[4 * i + 3]);
        }
        tc_fence_before();
        hand_back(a);
        __syncwarp();
        if (lane == 0) { __threadfence(); st_release_gpu(flag, 1u); }
        continue;
      }
      float pv[2][32];
      uint32_t* fix_flag = p.sk_flags + (blockIdx.x + G) * 4 + q;
      auto load_partial = [&](int c, float* dst) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float4 f = __ldcg(slot_ptr(blockIdx.x + G, c, i));
          dst[4 * i] = f.x; dst[4 * i + 1] = f.y; dst[4 * i + 2] = f.z; dst[4 * i + 3] = f.w;
        }
      };
      if (fixes) {
        // written about one kernel duration ago; fetched while the last K blocks of this tile are still running
        bool ok = lane == 0 ? gemm_flag_wait(fix_flag, 1u, gw, 6) : true;
        if (!__all_sync(0xffffffffu, ok)) break;
        load_partial(0, pv[0]);
      }
      // warp-uniform verdict: the tcgen05.ld below is a warp-wide instruction
      if (!__all_sync(0xffffffffu, gemm_wait(acc_full + a, (tile_i >> 1) & 1u, gw, 4))) break;
      tc_fence_after();
      bulk_wait_source_free<0>();   // this thread's previous pieces have left its staging row
      // 32 columns at a time, double-buffered: the load of chunk c + 1 is in flight while chunk c is quantised
      float v[2][32];
      tmem_ld32_issue(tbase, v[0]);
#pragma unroll
      for (int c = 0; c < BN / 32; c++) {
        tmem_ld_wait();
        if (c + 1 < BN / 32) tmem_ld32_issue(tbase + (c + 1) * 32, v[(c + 1) & 1]);
        float* vc = v[c & 1];
        if (fixes) {
          if (c + 1 < BN / 32) load_partial(c + 1, pv[(c + 1) & 1]);
          const float* pc = pv[c & 1];
#pragma unroll
          for (int i = 0; i < 32; i++) vc[i] = __fadd_rn(vc[i], pc[i]);
        }
        if (p.dbg_acc && row < p.M) {
          float4* dst = reinterpret_cast<float4*>(p.dbg_acc + (size_t)row * p.N + n0 + c * 32);
#pragma unroll
          for (int i = 0; i < 8; i++) dst[i] = make_float4(vc[4 * i], vc[4 * i + 1], vc[4 * i + 2], vc[4 * i + 3]);
        }
        uint4 qv;
        const uint32_t sf2 = encode_pair_f32<true>(vc, [&](float b0, float b1, float& m0, float& m1) {
          return pair_block_scales(b0, b1, p.inv_gs, m0, m1);
        }, qv);
        *reinterpret_cast<uint4*>(my_piece + 16 * c) = qv;
        *reinterpret_cast<uint16_t*>(my_piece + S::kValueB + 2 * c) = (uint16_t)sf2;
      }
      if (fixes) {
        __syncwarp();
        if (lane == 0) st_release_gpu(fix_flag, 0u);        // every lane has its partial in registers: the slot is free
      }
      tc_fence_before();
      hand_back(a);                 // 128 arrivals hand the accumulator back to the MMA warp
      fence_smem_to_async();
      if (row < p.M) {
        const size_t voff = (size_t)(n0 / 2), soff = (size_t)(p.N / 2 + n0 / 16);
        // one row piece to one destination row: the values by a bulk store; the scales by a bulk store when they are
        // a 16-byte granule (BN = 256), else (12 bytes at a 4-byte aligned offset) by three word stores from registers
        auto put = [&](char* dst) {
          bulk_store(dst + voff, my_piece, S::kValueB);
          if constexpr (S::kScaleB == 16) {
            bulk_store(dst + soff, my_piece + S::kValueB, 16);
          } else {
            const uint32_t* sw = reinterpret_cast<const uint32_t*>(my_piece + S::kValueB);
            uint32_t* dw = reinterpret_cast<uint32_t*>(dst + soff);
#pragma unroll
            for (int i = 0; i < S::kScaleB / 4; i++) dw[i] = sw[i];
          }
        };
        if (p.local_q) put(p.local_q + (size_t)row * qrow_bytes);
        if (p.nranks) {
          if (p.two_shot) {
            put(p.win[row % p.nranks] + buf_off + ((size_t)p.rank * p.capo + row / p.nranks) * kRecStride);
          } else {
            for (int d = 0; d < p.nranks; d++) put(p.win[d] + buf_off + ((size_t)p.rank * p.cap + row) * kRecStride);
          }
        }
      }
      bulk_commit();
      __syncwarp();
    }
    bulk_wait_done<0>();
  }
done:
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (leads && threadIdx.x == 0)
      for (uint32_t i = issued > (uint32_t)kStages ? issued - kStages : 0u; i < issued; i++) gemm_settle(full + i % kStages, (i / kStages) & 1u);
    if (!leads && threadIdx.x == 0)
      for (int w = 0; w < 2000; w++) __nanosleep(1000);     // its loads complete under the leader's barriers: 2 ms
    if (leads && threadIdx.x == 32) {
      if constexpr (G == 2) umma_commit_pair(settled); else umma_commit(settled);
      gemm_settle(settled, 0u);
    }
    __syncthreads();
  }
  if constexpr (G == 2) cluster_sync_all();   // neither CTA frees TMEM or leaves while the other's MMAs, commits or arrivals may still touch it
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    if constexpr (G == 2) tmem_dealloc_pair(tmem_base, kTmemCols); else tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Few rows (M <= 384): one narrow tile per CTA, its whole K loop in one CTA.
//
// Such a call streams the weights once, and what bounds it is the chain of ring stages: a stage of one K block of 64 takes a
// CTA 300 - 400 ns whatever the tile's width and rows, one of two about 600, one of four about 950.  So a stage holds up to
// four blocks, fetched by one copy per operand (the matrices are described as [K / 64][rows][64], a box of several blocks
// lands as consecutive swizzled tiles), and the tiles are narrow: 128 x BN, BN 64 (up to 128 rows), 96 or 128 columns, put a
// CTA on most of the SMs (N = 6144: 96, 128 or 144 of them), with a short set-up and a short epilogue that stores straight
// from registers.
// The K loop is NOT cut over CTAs (a cluster of four that sums its partials takes half as long at K = 8192): the FP32
// sums are then rounded elsewhere and about one value in 1e5 becomes another E2M1 value.  Whole chains give the accumulators
// of whole wide tiles bit for bit, so a row of such a call does not depend on the rows that share it.  (Above 384 rows it
// may: tiles that two CTAs share are sums of two chains, which those calls have always had.)
// Pushed rows leave as one 16-byte and one 2-byte store per 32 columns, straight from registers.  Wider packets cost more than
// they save where the window is in this GPU's memory (K = 1024, 64 / 200 / 384 rows to four ranks: 7.7 / 8.9 / 9.6 us; one bulk
// store a row 8.5 / 10.0 / 10.1; neighbouring lanes' stores through shared memory 7.9 / 9.5 / 9.7); over NVLink none of them
// has been timed.
// N = 6144, fresh weights for every call, us, 192- and 256-wide tiles -> these: M = 1: K = 1024 9.8 -> 7.2, K = 8192 48.6 -> 30.3;
// M = 64: K = 1024 10.6 -> 7.3, K = 2048 15.2 -> 10.7, K = 8192 44.4 -> 30.5; M = 128, K = 2048 15.3 -> 11.9; M = 200, K = 4096 26.7 -> 21.5;
// M = 300, K = 2048 16.5 -> 13.5; M = 384: K = 1024 11.6 -> 8.9, K = 4096 29.6 -> 22.5, K = 8192 48.9 -> 42.4.
// The A box holds only the valid rows, rounded up to eight: the MMA still takes 128 rows, and what it reads for the rest
// is the start of the B block or whatever follows it in shared memory, whose products land in accumulator rows that nobody
// reads.
constexpr int kNarrowStages = 16;
template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_narrow_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                   const __grid_constant__ GemmParams p) {
  static_assert(BN == 64 || BN == 96 || BN == 128, "tile width");
  constexpr int kBBytes = BN * kBK * 2;
  constexpr uint32_t kCols = BN == 64 ? 64 : 128;       // TMEM columns, a power of two
  constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int atoms = p.atoms, a_tile = p.a_rows * kBK * 2, a_bytes = atoms * a_tile, stage_bytes = a_bytes + atoms * kBBytes;
  const int stages = p.stages;
  // barriers beyond the 128 rows that the MMA reads from the last stage's last A tile
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + (stages - 1) * stage_bytes + max(stage_bytes, a_bytes - a_tile + kABytes));
  uint64_t* empty = full + kNarrowStages;
  uint64_t* acc_full = empty + kNarrowStages;
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_full + 1);
  volatile uint32_t* abort_flag = tmem_holder + 1;
  int issued = 0;                      // ring stages filled

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m_tiles = (p.M + kBM - 1) / kBM, kblocks = p.K / kBK, trips = (kblocks + atoms - 1) / atoms;
  // the tiles of one column range are neighbours: their weights cross HBM once
  const int m0 = (int)blockIdx.x % m_tiles * kBM, n0 = (int)blockIdx.x / m_tiles * BN;

  if (threadIdx.x == 32) { prefetch_tensormap(&map_a); prefetch_tensormap(&map_b); }
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; i++) { mbar_init(full + i, 1); mbar_init(empty + i, 1); }
    mbar_init(acc_full, 1);
    *abort_flag = 0u;
    mbar_init_fence();
  }
  if (warp == 1) { tmem_alloc(tmem_holder, kCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_holder;
  GemmWait gw{abort_flag, p.status, p.timeout_ns};

  pdl_wait_prior_grids();
  pdl_release_dependents();

  if (warp == 0) {
    if (lane == 0) {
      for (int st = 0, round = 0; issued < trips; issued++) {
        if (!gemm_wait(empty + st, (round & 1u) ^ 1u, gw, 1)) break;
        mbar_arrive_expect(full + st, stage_bytes);
        if (atoms > 1) {
          tma_load_3d(ring + st * stage_bytes, &map_a, m0, issued * atoms, full + st);
          tma_load_3d(ring + st * stage_bytes + a_bytes, &map_b, n0, issued * atoms, full + st);
        } else {
          tma_load_2d(ring + st * stage_bytes, &map_a, issued * kBK, m0, full + st);
          tma_load_2d(ring + st * stage_bytes + a_bytes, &map_b, issued * kBK, n0, full + st);
        }
        if (++st == stages) { st = 0; round++; }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      for (int it = 0, st = 0, round = 0; it < trips; it++) {
        if (!gemm_wait(full + st, round & 1u, gw, 3)) break;
        tc_fence_after();
        uint64_t da = umma_desc_k128(ring + st * stage_bytes), db = umma_desc_k128(ring + st * stage_bytes + a_bytes);
        const int n = min(atoms, kblocks - it * atoms);
        for (int j = 0; j < n; j++) {
#pragma unroll
          for (int k = 0; k < kBK / 16; k++)
            umma_bf16(tmem_base, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), kIdesc, (it | j | k) != 0 ? 1u : 0u);
          da += (uint64_t)(a_tile >> 4); db += (uint64_t)(kBBytes >> 4);
        }
        umma_commit(empty + st);
        if (++st == stages) { st = 0; round++; }
      }
      umma_commit(acc_full);
    }
  } else {
    const int q = warp & 3, row = m0 + q * 32 + lane;
    const bool good = __all_sync(0xffffffffu, gemm_wait(acc_full, 0u, gw, 4));
    tc_fence_after();
    if (good && !__any_sync(0xffffffffu, *abort_flag != 0u) && m0 + q * 32 < p.M) {
      const uint32_t tbase = tmem_base + ((uint32_t)(q * 32) << 16);
      const int qrow_bytes = p.N / 2 + p.N / 16;
      const size_t buf_off = p.nranks ? (size_t)(*p.call_counter & 1u) * p.buf_bytes : 0;
      float v[2][32];
      tmem_ld32_issue(tbase, v[0]);
#pragma unroll
      for (int c = 0; c < BN / 32; c++) {
        tmem_ld_wait();
        if (c + 1 < BN / 32) tmem_ld32_issue(tbase + (c + 1) * 32, v[(c + 1) & 1]);
        float* vc = v[c & 1];
        if (row < p.M) {
          if (p.dbg_acc) {
            float4* dst = reinterpret_cast<float4*>(p.dbg_acc + (size_t)row * p.N + n0 + c * 32);
#pragma unroll
            for (int i = 0; i < 8; i++) dst[i] = make_float4(vc[4 * i], vc[4 * i + 1], vc[4 * i + 2], vc[4 * i + 3]);
          }
          uint4 qv;
          const uint32_t sf2 = encode_pair_f32<true>(vc, [&](float b0, float b1, float& m0_, float& m1_) {
            return pair_block_scales(b0, b1, p.inv_gs, m0_, m1_);
          }, qv);
          const size_t voff = (size_t)(n0 / 2 + 16 * c), soff = (size_t)(p.N / 2 + n0 / 16 + 2 * c);
          auto put = [&](char* dst) {
            *reinterpret_cast<uint4*>(dst + voff) = qv;
            *reinterpret_cast<uint16_t*>(dst + soff) = (uint16_t)sf2;
          };
          if (p.local_q) put(p.local_q + (size_t)row * qrow_bytes);
          if (p.nranks) {
            if (p.two_shot) put(p.win[row % p.nranks] + buf_off + ((size_t)p.rank * p.capo + row / p.nranks) * kRecStride);
            else for (int d = 0; d < p.nranks; d++) put(p.win[d] + buf_off + ((size_t)p.rank * p.cap + row) * kRecStride);
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0u) {
    if (threadIdx.x == 0)
      for (int i = max(0, issued - stages); i < issued; i++) gemm_settle(full + i % stages, (i / stages) & 1);
    if (threadIdx.x == 32) gemm_settle(acc_full, 0u);       // committed behind every MMA issued
    __syncthreads();
  }
  if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem_base, kCols); }
}

// ---- host side ----
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}
static bool make_map(CUtensorMap* m, const void* base, int rows, int k, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)k * 2};
  cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same matrix as [K / 64][rows][64]: one box covers `atoms` K blocks.
static bool make_map_3d(CUtensorMap* m, const void* base, int rows, int k, int box_rows, int atoms) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {(cuuint64_t)kBK, (cuuint64_t)rows, (cuuint64_t)(k / kBK)};
  cuuint64_t strides[2] = {(cuuint64_t)k * 2, (cuuint64_t)kBK * 2};
  cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, (cuuint32_t)atoms};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Zeroed device memory, also while a stream of this thread is being captured (the allocation is not part of the graph).
static void* alloc_zeroed(size_t bytes) {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return nullptr;
  void* p = nullptr;
  cudaStream_t s = nullptr;
  bool ok = cudaMalloc(&p, bytes) == cudaSuccess && cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMemsetAsync(p, 0, bytes, s) == cudaSuccess && cudaStreamSynchronize(s) == cudaSuccess;
  if (s) cudaStreamDestroy(s);
  if (!ok) {
    cudaGetLastError();
    if (p) cudaFree(p);
    p = nullptr;
  }
  cudaThreadExchangeStreamCaptureMode(&mode);
  return p;
}

// The status block of a device, allocated by the first thread that needs it.
static StatusWords* gemm_status_word() {
  static std::atomic<StatusWords*> words[64];
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
  StatusWords* p = words[dev].load(std::memory_order_acquire);
  if (!p) {
    std::lock_guard<std::mutex> g(mu);
    p = words[dev].load(std::memory_order_acquire);
    if (!p) {
      p = (StatusWords*)alloc_zeroed(sizeof(StatusWords));
      words[dev].store(p, std::memory_order_release);
    }
  }
  return p;
}

// Workspaces of the stream-K split: one slot of 128 x 256 floats and four flags per SM (19 MB on a B200).  A flag says that
// a partial is there, not whose it is, so two launches that may run at the same time never share a workspace:
//   - the launches of a stream follow one another and share one (streams are told apart by their id, which is never used
//     again).  The first kSpaces streams of a device have their own; the launches of all later ones take turns on one
//     more, by an event;
//   - the launches that one capture records on one stream share one that their graph owns: the replays of a graph follow
//     one another.  It can serve another graph once that one and its instances are gone.
// Memory is allocated when it is first needed and kept; fp4ar_gemm_reset gives back what no graph owns.
struct StreamKSpace {
  void* mem = nullptr;                   // partials, then flags
  unsigned long long stream = 0, capture = 0;
  bool graph_owned = false;
  std::atomic<bool> idle{false};         // set when the owning graph is gone, from a thread of CUDA: nothing else happens there
};
struct StreamKPool {
  std::vector<std::unique_ptr<StreamKSpace>> spaces;
  std::unique_ptr<StreamKSpace> shared;  // of the streams beyond kSpaces
  cudaEvent_t turn = nullptr;            // its last launch
};
constexpr int kSpaces = 8;
static StreamKPool* const g_stream_k = new StreamKPool[64];      // never destroyed: a graph may be released while the process ends
static std::mutex g_stream_k_mu;
static size_t stream_k_partial_bytes() { return (size_t)device_sm_count() * kBM * 256 * sizeof(float); }
static size_t stream_k_flag_bytes() { return (size_t)device_sm_count() * 4 * sizeof(uint32_t); }

// The workspace of one launch, held until the launch is enqueued.
class StreamKLease {
 public:
  explicit StreamKLease(cudaStream_t stream) : lock_(g_stream_k_mu), stream_(stream) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return;
    StreamKPool& pool = g_stream_k[dev];
    cudaStreamCaptureStatus status;
    unsigned long long id = 0, capture = 0;
    cudaGraph_t graph = nullptr;
    if (cudaStreamGetCaptureInfo(stream, &status, &capture, &graph) != cudaSuccess) { cudaGetLastError(); return; }
    const bool recording = status == cudaStreamCaptureStatusActive;
    if (recording) id = (unsigned long long)(uintptr_t)stream;             // the id cannot be asked for during a capture
    else if (status != cudaStreamCaptureStatusNone || cudaStreamGetId(stream, &id) != cudaSuccess) { cudaGetLastError(); return; }
    StreamKSpace* free_one = nullptr;
    int streams = 0;
    for (auto& s : pool.spaces) {
      if (s->graph_owned && s->idle.load(std::memory_order_acquire)) free_one = s.get();
      else if (s->graph_owned == recording && s->stream == id && (!recording || s->capture == capture)) { space_ = s.get(); return; }
      else if (!s->graph_owned) streams++;
    }
    if (recording) {
      StreamKSpace* s = free_one ? free_one : add(pool);
      if (!s || !zero_flags(s) || !give_to(graph, s)) return;
      s->stream = id; s->capture = capture;
      space_ = s;
    } else if (streams < kSpaces) {
      StreamKSpace* s = add(pool);
      if (!s) return;
      s->stream = id;
      space_ = s;
    } else {
      if (!pool.turn && cudaEventCreateWithFlags(&pool.turn, cudaEventDisableTiming) != cudaSuccess) { cudaGetLastError(); return; }
      if (!pool.shared) pool.shared = make();
      if (!pool.shared || cudaStreamWaitEvent(stream, pool.turn, 0) != cudaSuccess) { cudaGetLastError(); return; }
      space_ = pool.shared.get();
      turn_ = pool.turn;
    }
  }
  ~StreamKLease() {
    if (turn_ && cudaEventRecord(turn_, stream_) != cudaSuccess) cudaGetLastError();
  }
  explicit operator bool() const { return space_ != nullptr; }
  float* partial() const { return (float*)space_->mem; }
  uint32_t* flags() const { return (uint32_t*)((char*)space_->mem + stream_k_partial_bytes()); }

 private:
  static std::unique_ptr<StreamKSpace> make() {
    std::unique_ptr<StreamKSpace> s(new StreamKSpace);
    s->mem = alloc_zeroed(stream_k_partial_bytes() + stream_k_flag_bytes());
    if (!s->mem) s.reset();
    return s;
  }
  static StreamKSpace* add(StreamKPool& pool) {
    auto s = make();
    if (!s) return nullptr;
    pool.spaces.push_back(std::move(s));
    return pool.spaces.back().get();
  }
  // A graph that ended in a launch which gave up may have left flags behind.
  static bool zero_flags(StreamKSpace* s) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return false;
    cudaStream_t st = nullptr;
    const bool ok = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
                    cudaMemsetAsync((char*)s->mem + stream_k_partial_bytes(), 0, stream_k_flag_bytes(), st) == cudaSuccess &&
                    cudaStreamSynchronize(st) == cudaSuccess;
    if (st) cudaStreamDestroy(st);
    if (!ok) cudaGetLastError();
    cudaThreadExchangeStreamCaptureMode(&mode);
    return ok;
  }
  static void CUDART_CB released(void* p) { static_cast<StreamKSpace*>(p)->idle.store(true, std::memory_order_release); }
  static bool give_to(cudaGraph_t graph, StreamKSpace* s) {
    s->graph_owned = true;
    s->idle.store(false, std::memory_order_release);
    cudaUserObject_t object;
    if (cudaUserObjectCreate(&object, s, released, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
      cudaGetLastError();
      s->idle.store(true, std::memory_order_release);
      return false;
    }
    if (cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove) == cudaSuccess) return true;
    cudaGetLastError();
    cudaUserObjectRelease(object, 1);
    return false;
  }
  std::lock_guard<std::mutex> lock_;
  cudaStream_t stream_;
  StreamKSpace* space_ = nullptr;
  cudaEvent_t turn_ = nullptr;
};

}  // namespace fp4ar

using namespace fp4ar;

// Which shape a call takes.  `units` = CTAs (or CTA pairs) that work, `tiles` = output tiles of that shape.
struct GemmPlan { int pair, bn, stream_k, units, tiles, narrow; };
static GemmPlan plan_gemm(int M, int N, int K, int sms, bool env) {
  // Tile width of single CTAs: the one whose tiles keep the persistent CTAs busier over all waves.  A 192-wide tile was
  // measured at about 0.87 of the per-cycle work of a 256-wide one (M = 4096: 321 vs 315 us at K = 8192 although its
  // last wave is full), so it is only taken where it wins clearly (M = 1024: 111 vs 123 us); N must be a multiple of
  // 192 too.  FP4AR_GEMM_TILE_N = 192 / 256 forces it (and single CTAs).
  int bn = 256;
  bool stream_k = false, pair = false;
  // Few rows: one narrow tile per CTA (see gemm_narrow_kernel), the widest of 128, 96 and 64 columns that gives two
  // thirds of the SMs a tile and none of them two.  An environment override of the shapes below switches it off.
  if (!(env && (std::getenv("FP4AR_GEMM_TILE_N") || std::getenv("FP4AR_GEMM_STREAM_K") || std::getenv("FP4AR_GEMM_PAIR"))) && M <= 384) {
    for (int w : {128, 96, 64}) {
      const int t = N / w * ((M + kBM - 1) / kBM);
      if (N % w == 0 && (3 * t >= 2 * sms || w == 64) && t <= sms) return GemmPlan{0, w, 0, t, t, 1};
    }
  }
  const char* force = env ? std::getenv("FP4AR_GEMM_TILE_N") : nullptr;
  const char* fsk = env ? std::getenv("FP4AR_GEMM_STREAM_K") : nullptr;
  const char* fp = env ? std::getenv("FP4AR_GEMM_PAIR") : nullptr;
  auto busy = [&](int w) {
    const long tiles = (long)(N / w) * ((M + kBM - 1) / kBM);
    return (double)tiles / (double)(((tiles + sms - 1) / sms) * sms);
  };
  if (N % 192 == 0 && 0.80 * busy(192) > busy(256)) bn = 192;
  if (force && std::atoi(force) == 256) bn = 256;
  if (force && std::atoi(force) == 192 && N % 192 == 0) bn = 192;
  // Stream-K (256-wide tiles, the K loop cut into equal ranges per CTA) where whole tiles would leave the last wave
  // of CTAs partly idle and the K loop is long enough to pay for the partial sums (K = 2048: 36.9 us against 33.0 us
  // with whole 192-wide tiles at M = 1024, level at M = 2048, 77.8 against 79.9 at M = 4096; K = 8192: 86 / 143 /
  // 264 us against 96 / 154 / 296 at M = 1024 / 2048 / 4096); FP4AR_GEMM_STREAM_K = 0 / 1 overrides.
  const long tiles256 = (long)(N / 256) * ((M + kBM - 1) / kBM);
  stream_k = tiles256 > sms && tiles256 % sms != 0 && busy(256) < 0.95 && (K >= 4096 || tiles256 >= 4 * sms) &&
             !(force && std::atoi(force) == 192);
  if (fsk) stream_k = std::atoi(fsk) != 0 && tiles256 > sms && tiles256 % sms != 0;
  if (stream_k) bn = 256;
  // CTA pairs (tcgen05 cta_group::2) where the K loop is long or there are many tiles: measured against single CTAs
  // at M = 1024 / 2048 / 4096 / 16384: K = 8192: 80 / 131 / 252 / 1054 us against 88 / 143 / 268 / 1078; K = 4096:
  // 52 / 76 / 135 / 506 against 53 / 78 / 137 / 524; K = 2048: 35 / 49 / 80 / 260 against 33 / 47 / 78 / 266.
  // FP4AR_GEMM_PAIR = 0 / 1 overrides.
  const bool want_pair = fp ? std::atoi(fp) != 0 : ((K >= 4096 || M >= 8192) && !force);
  long tiles = (long)(N / bn) * ((M + kBM - 1) / kBM);
  int units = sms;
  if (want_pair && sms >= 2) {
    pair = true; bn = 256;
    units = sms / 2;
    tiles = (long)(N / 256) * ((M + 2 * kBM - 1) / (2 * kBM));
    const double busy2 = (double)tiles / (double)(((tiles + units - 1) / units) * units);
    stream_k = tiles > units && tiles % units != 0 && busy2 < 0.95 && (K >= 4096 || tiles >= 4 * units);
    if (fsk) stream_k = std::atoi(fsk) != 0 && tiles > units && tiles % units != 0;
  }
  if (tiles < units) units = (int)tiles;
  return GemmPlan{pair ? 1 : 0, bn, stream_k ? 1 : 0, units, (int)tiles, 0};
}

template <int BN, int G>
static int launch_gemm(const CUtensorMap& ma, const CUtensorMap& mb, GemmParams p, cudaStream_t stream) {
  using S = GemmShape<BN, G>;
  // The shared-memory limit and the number of resident pairs are set / asked once per device, not on every launch.
  static std::atomic<int> resident[64];          // 0: not asked yet; units (CTAs or pairs) that can be resident together
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cuda_fail();
  int fits = resident[dev].load(std::memory_order_acquire);
  if (!fits && cudaFuncSetAttribute(gemm_nvfp4_kernel<BN, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem) != cudaSuccess)
    return cuda_fail();
  const int tiles = (p.N / BN) * ((p.M + kBM * G - 1) / (kBM * G));
  const int sms = device_sm_count();
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.dynamicSmemBytes = S::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  int units = sms / G;
  cfg.attrs = attr;
  if (G == 2) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(sms & ~1);
    // pairs that can be resident together: the grid is persistent, every pair must be
    if (!fits && (cudaOccupancyMaxActiveClusters(&fits, gemm_nvfp4_kernel<BN, G>, &cfg) != cudaSuccess || fits < 1)) return cuda_fail();
    if (fits < units) units = fits;
  }
  resident[dev].store(G == 2 ? fits : units, std::memory_order_release);     // every thread computes the same value
  // Programmatic dependent launch: a CTA may start (barrier set-up, TMEM allocation) on an SM that the previous
  // kernel's CTA has left while other CTAs of that kernel still run; it touches global memory only after
  // griddepcontrol.wait.  FP4AR_GEMM_PDL = 0 turns it off.
  {
    const char* e = std::getenv("FP4AR_GEMM_PDL");
    if (!e || std::atoi(e) != 0) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
      cfg.numAttrs++;
    }
  }
  if (tiles < units) units = tiles;
  if (p.stream_k && (tiles <= units || tiles % units == 0)) p.stream_k = 0;      // fewer units fit than planned: whole tiles (see SegIter)
  cfg.gridDim = dim3(units * G);
  if (cudaLaunchKernelEx(&cfg, gemm_nvfp4_kernel<BN, G>, ma, mb, p) != cudaSuccess) return cuda_fail();
  return cuda_check_launch();
}

template <int BN>
static int launch_narrow(const CUtensorMap& ma, const CUtensorMap& mb, GemmParams p, int tiles, cudaStream_t stream) {
  const int a_tile = p.a_rows * kBK * 2, stage = p.atoms * (a_tile + BN * kBK * 2);
  const int last = (p.atoms - 1) * a_tile + kABytes, pad = stage < last ? last - stage : 0;     // what the MMA reads as A
  const int tail = 512 + 1024;                          // barriers, alignment slack
  constexpr int kWhole = 224 * 1024;
  p.stages = (kWhole - tail - pad) / stage;
  if (p.stages > kNarrowStages) p.stages = kNarrowStages;
  const int trips = (p.K / kBK + p.atoms - 1) / p.atoms;
  if (p.stages > trips) p.stages = trips;               // a short K loop leaves room for the next launch's CTAs
  const int smem = p.stages * stage + pad + tail;
  static std::atomic<int> raised[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cuda_fail();
  if (!raised[dev].load(std::memory_order_acquire)) {
    if (cudaFuncSetAttribute(gemm_narrow_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWhole) != cudaSuccess) return cuda_fail();
    raised[dev].store(1, std::memory_order_release);
  }
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.blockDim = dim3(kGemmThreads);
  cfg.gridDim = dim3(tiles);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  const char* e = std::getenv("FP4AR_GEMM_PDL");
  cfg.numAttrs = e && std::atoi(e) == 0 ? 0 : 1;
  if (cudaLaunchKernelEx(&cfg, gemm_narrow_kernel<BN>, ma, mb, p) != cudaSuccess) return cuda_fail();
  return cuda_check_launch();
}

extern "C" int fp4ar_gemm_nvfp4(const fp4ar_push_view* push, int two_shot, const void* x, const void* wt, int M, int N,
                                int K, float gs, void* local_q, float* dbg_acc, fp4ar_stream stream) {
  if (!x || !wt || M < 1 || N < 256 || K < kBK || (N % 256) || (K % kBK) || !(gs > 0.0f)) return FP4AR_ERR_ARGUMENT;
  if (((uintptr_t)x | (uintptr_t)wt | (uintptr_t)local_q | (uintptr_t)dbg_acc) & 15) return FP4AR_ERR_ARGUMENT;
  if (!push && !local_q && !dbg_acc) return FP4AR_ERR_ARGUMENT;
  const GemmPlan pl = plan_gemm(M, N, K, device_sm_count(), /*env=*/true);
  const int bn = pl.bn;
  const bool stream_k = pl.stream_k != 0, pair = pl.pair != 0;
  GemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K; p.inv_gs = 1.0f / gs;
  p.local_q = (char*)local_q; p.dbg_acc = dbg_acc;
  if (push) {
    if (N != FP4AR_HIDDEN || push->nranks < 1 || push->nranks > FP4AR_MAX_RANKS || !push->call_counter) return FP4AR_ERR_ARGUMENT;
    if (M > push->cap) return FP4AR_ERR_ARGUMENT;
    p.nranks = push->nranks; p.rank = push->rank; p.cap = push->cap; p.capo = push->capo;
    p.buf_bytes = push->buffer_bytes; p.call_counter = push->call_counter; p.two_shot = two_shot ? 1 : 0;
    for (int r = 0; r < push->nranks; r++) {
      if (!push->windows[r]) return FP4AR_ERR_ARGUMENT;
      p.win[r] = (char*)push->windows[r];
    }
    // host-side bound of the farthest byte this call can touch in a window
    const size_t last = two_shot ? ((size_t)(p.nranks - 1) * p.capo + (size_t)(M - 1) / p.nranks + 1) * kRecStride
                                 : ((size_t)(p.nranks - 1) * p.cap + (size_t)M) * kRecStride;
    if (last > p.buf_bytes) return FP4AR_ERR_ARGUMENT;
  }
  p.status = gemm_status_word();
  if (!p.status) return cuda_fail();
  p.timeout_ns = 2000000000ull;
  std::optional<StreamKLease> lease;
  if (stream_k) {
    lease.emplace((cudaStream_t)stream);
    if (*lease) { p.stream_k = 1; p.sk_partial = lease->partial(); p.sk_flags = lease->flags(); }
  }
  CUtensorMap ma, mb;
  if (pl.narrow) {
    p.a_rows = M < kBM ? (M + 7) / 8 * 8 : kBM;
    // K blocks per stage: as many, up to four, as leave the ring two stages (M = 64, K = 8192: 30.5 us; four shorter stages took 38)
    p.atoms = 4;
    while (p.atoms > 1 && (p.atoms > K / kBK || p.atoms * (p.a_rows + bn) * kBK * 2 > 100 * 1024)) p.atoms /= 2;
    const bool maps = p.atoms > 1 ? make_map_3d(&ma, x, M, K, p.a_rows, p.atoms) && make_map_3d(&mb, wt, N, K, bn, p.atoms)
                                  : make_map(&ma, x, M, K, p.a_rows) && make_map(&mb, wt, N, K, bn);
    if (!maps) return FP4AR_ERR_UNSUPPORTED;
    if (bn == 64) return launch_narrow<64>(ma, mb, p, pl.tiles, (cudaStream_t)stream);
    return bn == 96 ? launch_narrow<96>(ma, mb, p, pl.tiles, (cudaStream_t)stream)
                    : launch_narrow<128>(ma, mb, p, pl.tiles, (cudaStream_t)stream);
  }
  if (!make_map(&ma, x, M, K, kBM) || !make_map(&mb, wt, N, K, pair ? bn / 2 : bn)) return FP4AR_ERR_UNSUPPORTED;
  if (pair) return launch_gemm<256, 2>(ma, mb, p, (cudaStream_t)stream);
  return bn == 192 ? launch_gemm<192, 1>(ma, mb, p, (cudaStream_t)stream) : launch_gemm<256, 1>(ma, mb, p, (cudaStream_t)stream);
}

// The schedule of one launch, computed on the host with the kernel's own iterator (for tests and tools): which shape
// a call of this size takes, and the segments of one unit as (tile, first K block, K blocks, kind) quadruples.
extern "C" int fp4ar_gemm_plan(int M, int N, int K, int sms, int* pair, int* tile_n, int* stream_k, int* units, int* tiles,
                               int unit, int* segments, int max_segments) {
  if (M < 1 || N < 256 || K < kBK || (N % 256) || (K % kBK) || sms < 2 || !pair || !tile_n || !stream_k || !units || !tiles)
    return -1;
  GemmPlan pl = plan_gemm(M, N, K, sms, /*env=*/false);
  *pair = pl.pair; *tile_n = pl.bn; *stream_k = pl.stream_k; *units = pl.units; *tiles = pl.tiles;
  if (!segments) return 0;
  if (unit < 0 || unit >= pl.units) return -1;
  SegIter it(pl.stream_k, pl.tiles, K / kBK, unit, pl.units);
  Seg sg;
  int n = 0;
  while (it.next(sg)) {
    if (n < max_segments) { segments[4 * n] = sg.tile; segments[4 * n + 1] = sg.lo; segments[4 * n + 2] = sg.count; segments[4 * n + 3] = sg.kind; }
    n++;
  }
  return n;
}

extern "C" int fp4ar_gemm_reset(void) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cuda_fail();
  if (cudaDeviceSynchronize() != cudaSuccess) return cuda_fail();
  StatusWords* s = gemm_status_word();
  if (!s) return cuda_fail();
  if (cudaMemset(s, 0, sizeof(StatusWords)) != cudaSuccess) return cuda_fail();
  std::lock_guard<std::mutex> g(g_stream_k_mu);
  if (cudaDeviceSynchronize() != cudaSuccess) return cuda_fail();     // what was enqueued before the lock was taken
  StreamKPool& pool = g_stream_k[dev];
  auto in_use = [](const StreamKSpace& s) { return s.graph_owned && !s.idle.load(std::memory_order_acquire); };
  for (auto& s : pool.spaces)
    if (in_use(*s) && cudaMemset((char*)s->mem + stream_k_partial_bytes(), 0, stream_k_flag_bytes()) != cudaSuccess) return cuda_fail();
  std::vector<std::unique_ptr<StreamKSpace>> kept;
  for (auto& s : pool.spaces) {
    if (in_use(*s)) kept.push_back(std::move(s));
    else cudaFree(s->mem);
  }
  pool.spaces.swap(kept);
  if (pool.shared) { cudaFree(pool.shared->mem); pool.shared.reset(); }
  if (cudaDeviceSynchronize() != cudaSuccess) return cuda_fail();
  return FP4AR_OK;
}

extern "C" const void* fp4ar_gemm_workspace(fp4ar_stream stream) {
  const StreamKLease lease((cudaStream_t)stream);
  return lease ? lease.partial() : nullptr;
}

extern "C" int fp4ar_gemm_status(fp4ar_status_words* out) {
  StatusWords* s = gemm_status_word();
  if (!s || !out) return FP4AR_ERR_ARGUMENT;
  if (cudaMemcpy(out, s, sizeof(StatusWords), cudaMemcpyDeviceToHost) != cudaSuccess) return cuda_fail();
  return FP4AR_OK;
}
