// Dense and grouped block-scaled FP8 GEMM for sm_100a with fp32 scales:
//   out = cast( sum_kb (A_kb * B_kb^T) * sa[:,kb] * sb[nb,kb] ).
//
// Stands in for the reference's fp8_blockwise_scaled_mm
// (sgl-kernel/csrc/gemm/fp8_blockwise_gemm_kernel.cu:165-423), the Triton kernel
// _w8a8_block_fp8_matmul (python/sglang/srt/layers/quantization/fp8_kernel.py:493-575) and, grouped,
// fp8_blockwise_scaled_grouped_mm (sgl-kernel/csrc/moe/fp8_blockwise_moe_kernel.cu).
//
// The fp32 scales differ per row and per k-block, so partial sums cannot be chained inside the tensor core: every
// k-block's product is read out of tensor memory and promoted into fp32 registers.  Per 128 x 256 x 128 k-block that is
// 512 cycles of tensor pipe beside 362 cycles of tensor-memory loads and packed FMAs (each measured alone and together),
// so the read-out fits under the MMAs as long as nothing makes either side wait.  One persistent CTA per SM, 12 warps:
//   warps 0-7   promotion + epilogue: each owns 32 rows (its tensor-memory lane quadrant) x half of the tile's columns;
//               per k-block it reads the partial sums with tcgen05.ld in 64-column chunks, hands the accumulator back
//               after the last chunk has landed, and does acc += partial * (sa[m,kb] * sb[nb,kb]) with packed FMAs
//   TMA warp    producer: one A box (128 x 128 B) and one or two B boxes per k-block into a 4-stage ring, 128-byte swizzle
//   MMA warp    issuer: 4 x tcgen05.mma kind::f8f6f4 (M128 x N256 x K32) per k-block into one of two accumulators, each
//               started fresh per k-block; one commit per k-block signals "stage reusable" and "partial sums ready"
//   stager warp copies the scales of four k-blocks per ring slot with cp.async, up to 24 k-blocks ahead
// What the read-out loop must not do, each measured on [4096, 7168] x [36864, 7168] (1240-1320 us before, 975 us now, in
// cycles per k-block 1300 -> 800; the same results to the bit):
//   * go through generic pointers: pointers into aligned dynamic shared memory cost the slow load path and 64-bit address
//     arithmetic in every barrier operation (1147 -> 977); all shared addresses are 32-bit integers here;
//   * wait for its scale: products staged by a warp that loads, multiplies and stores one slot at a time paced the kernel
//     at one slot per global-memory round trip (1300), and a scale fetched where it is used costs its latency (977 -> 863);
//   * spill: shared memory takes the whole L1, so a spilled register is an L2 round trip.  Eight warps of 128 columns with
//     216 registers hold the accumulators and a 64-column chunk; sixteen warps of 64 columns (104 registers) spill;
//   * write its row in 16-byte pieces (863 -> 803 with 32-byte stores).
// What bounds it now is the chain of waits in the read-out warps: 803 cycles per k-block (739 without the stores) where the
// MMAs need 512, as many on zeros as on random data.  Power only sets the clock that they run at: at large M 1.45 GHz on
// random data and 1.965 GHz on zeros (1050 and 784 us for the product above).  (A CTA pair with two 128-column halves and
// four accumulators measured 946 cycles without loads or scales: the accumulator's round trip crosses the cluster.)
// All mbarrier waits are bounded; a wait that gives up records a code in a device status word and every role drains to
// a common exit where tensor memory is released.
#include <algorithm>

#include "gemm_common.cuh"

namespace b200 {
namespace {

constexpr int TILE_M = 128;
constexpr int BLOCK_K = 128;
constexpr int kTmemCols = 512;
constexpr int kGroupM = 32;     // 128-row blocks per rasterisation group: the group's A rows (<= 4096 x K bytes) stay in
                                // L2 while every weight slice is streamed once per group
constexpr int kScaleGroup = 4;  // k-blocks per scale-ring slot
constexpr int kScaleSlots = 6;  // the stager runs up to 24 k-blocks ahead
constexpr int kStages = 4;
constexpr int kABytes = TILE_M * BLOCK_K;
constexpr int kBHalfBytes = 128 * BLOCK_K;      // the weight rows of one 128-column half
constexpr int kBBytes = 2 * kBHalfBytes;
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kEpiWarps = 8;
constexpr int kTmaWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1, kStagerWarp = kEpiWarps + 2;
constexpr int kThreads = 32 * (kEpiWarps + 4);
constexpr int kReleaseThreads = 32 * (kEpiWarps + 2);   // TMA warp, MMA warp, read-out warps (pdl_release)
constexpr int CPW = 128;        // columns per read-out warp: one half of the tile
constexpr int kChunk = 64;      // columns per tensor-memory round trip (32: up to 4 % slower from 512 rows on)
constexpr int kSlotFloats = TILE_M * kScaleGroup + 2 * kScaleGroup;   // [128 rows][4 k-blocks], then [2 halves][4]
constexpr int kScaleBytes = kScaleSlots * kSlotFloats * 4;
constexpr int kMaxExperts = 1024;               // grouped form: m-tile prefix table in shared memory
constexpr int kSmemBytes = kStages * kStageBytes + kScaleBytes + 1024 /*alignment slack*/ + 512 /*barriers*/;
static_assert(kSmemBytes + (kMaxExperts + 2) * 4 <= 227 * 1024, "shared memory");
// The launch gives every thread 168 registers (12 warps); the helper warpgroup hands 96 per thread back and the read-out
// warps take 48 more each: 128 accumulators, a 64-column chunk and the loop without a spill (208 spills).  setmaxnreg.inc
// WAITS until the CTA's pool holds the registers it asks for, so the request must never exceed what the helpers release
// (the build checks the register count ptxas reports).
constexpr int kLaunchRegs = 168, kEpiRegs = 216, kHelperRegs = 72;
static_assert(kEpiWarps * (kEpiRegs - kLaunchRegs) <= 4 * (kLaunchRegs - kHelperRegs),
              "read-out warps would wait forever for registers nobody releases");

__device__ __forceinline__ void tile_coords(int tile, int m_blocks, int n_blocks, int& m_blk, int& n_blk) {
  const int group_size = kGroupM * n_blocks;
  const int group = tile / group_size;
  const int first_m = group * kGroupM;
  const int rows = min(kGroupM, m_blocks - first_m);
  const int in_group = tile - group * group_size;
  m_blk = first_m + in_group % rows;
  n_blk = in_group / rows;
}

// Where a tile lives.  Dense: tiles of the [M, N] output, rasterised in groups of kGroupM row blocks.
// Grouped: the row tiles of all experts laid end to end (tile_m_start[e] = first row tile of expert e,
// in shared memory), n-blocks fastest so that neighbouring CTAs stream different slices of the same
// expert's weights while sharing its few activation rows through L2.
struct TileInfo {
  int row0;        // first row of A / out of the tile
  int valid_rows;  // rows of the tile that belong to the problem (<= TILE_M)
  int n0;          // first output column
  int b_row0;      // first row of the [E*N, K] weight matrix
  int expert;
  int halves;      // 128-column halves that hold output columns (1 or 2)
};

template <bool GROUPED>
__device__ __forceinline__ TileInfo get_tile(int tile, const GemmParams& p, int m_blocks, int n_blocks,
                                             const int* tile_m_start) {
  TileInfo t;
  int n_blk;
  if constexpr (!GROUPED) {
    int m_blk;
    tile_coords(tile, m_blocks, n_blocks, m_blk, n_blk);
    t.row0 = m_blk * TILE_M;
    t.valid_rows = min(TILE_M, p.M - t.row0);
    t.n0 = n_blk * p.tile_n;
    t.b_row0 = t.n0;
    t.expert = 0;
  } else {
    const int mt = tile / n_blocks;
    n_blk = tile - mt * n_blocks;
    int lo = 0, hi = p.num_experts;   // last e with tile_m_start[e] <= mt
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile_m_start[mid] <= mt) lo = mid; else hi = mid;
    }
    t.expert = lo;
    const int m_blk = mt - tile_m_start[lo];
    const int m_e = p.problem_sizes[lo * 3];
    // Tables that do not describe the buffers (left over from another batch, never filled) must not send a
    // store outside `out`: the tile is clamped into [0, total rows).
    t.row0 = min(max(p.expert_offsets[lo] + m_blk * TILE_M, 0), p.M - 1);
    t.valid_rows = max(0, min(min(TILE_M, m_e - m_blk * TILE_M), p.M - t.row0));
    t.n0 = n_blk * p.tile_n;
    t.b_row0 = lo * p.N + t.n0;
  }
  t.halves = (p.tile_n == 256 && p.N - t.n0 > 128) ? 2 : 1;
  return t;
}

// One unit of a CTA's work list: a whole tile, or one split of a tile's k-blocks.
struct Work {
  int tile, split, kb_begin, kb_end;
  bool partial;   // the result is a partial sum for the workspace, not an output tile
};
__device__ __forceinline__ Work decode_work(int vt, const GemmParams& p, int nkb, bool grouped) {
  if (grouped || p.split_k == 1) return Work{vt, 0, 0, nkb, false};
  if (vt < p.tail_first) return Work{vt, 0, 0, nkb, false};
  const int r = vt - p.tail_first;
  const int tile = p.tail_first + r / p.split_k, split = r % p.split_k;
  const int kb0 = split * p.kb_per_split;
  return Work{tile, split, kb0, min(nkb, kb0 + p.kb_per_split), true};
}

template <bool GROUPED, typename OutT>
__global__ void __launch_bounds__(kThreads, 1)
gemm_block_fp8_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                      const GemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  // 1024-byte alignment: the 128-byte swizzle pattern is a function of address bits [4,10).
  const uint32_t smem_a = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t smem_b = smem_a + kStages * kABytes;
  const uint32_t smem_scale = smem_a + kStages * kStageBytes;
  const uint32_t full_bar = smem_scale + kScaleBytes;         // operands of the stage have landed
  const uint32_t done_bar = full_bar + 8 * kStages;           // the k-block's MMAs completed
  const uint32_t acc_empty = done_bar + 8 * kStages;          // accumulator has been read out
  const uint32_t scale_full = acc_empty + 8 * 2;              // scale-ring slot written
  const uint32_t scale_empty = scale_full + 8 * kScaleSlots;
  __shared__ uint32_t tmem_slot;
  __shared__ int tile_m_start[GROUPED ? kMaxExperts + 1 : 1];

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int m_blocks = (p.M + TILE_M - 1) / TILE_M;
  const int n_blocks = (p.N + p.tile_n - 1) / p.tile_n;
  const int nkb = (p.K + BLOCK_K - 1) / BLOCK_K;

  if constexpr (GROUPED) {
    pdl_wait();     // the tables come from the kernels before this one
    build_tile_table(tile_m_start, p.problem_sizes, p.num_experts, TILE_M);
  }

  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      sa::init(full_bar + 8 * i, 1);
      sa::init(done_bar + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) sa::init(acc_empty + 8 * i, kEpiWarps);
    for (int i = 0; i < kScaleSlots; ++i) {
      sa::init(scale_full + 8 * i, 32);         // every lane of the stager warp
      sa::init(scale_empty + 8 * i, kEpiWarps);
    }
    fence_mbar_init();
    fence_proxy_async_smem();
  }
  if (warp == kTmaWarp && lane == 0) {
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_b);
  }
  if (warp == kMmaWarp) {
    tmem_alloc(&tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
  const int num_tiles = GROUPED ? tile_m_start[p.num_experts] * n_blocks : m_blocks * n_blocks;
  // split-K: every tile from tail_first on becomes split_k work units (split fastest), each covering
  // kb_per_split k-blocks; tail_first = 0 splits all tiles, otherwise only the last wave
  const int split_k = GROUPED ? 1 : p.split_k;
  const int tail_first = (GROUPED || split_k == 1) ? num_tiles : p.tail_first;
  const int num_vtiles = tail_first + (num_tiles - tail_first) * split_k;

  if (warp >= kEpiWarps) {
  // ====================================================================== helper warpgroup
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kHelperRegs));
  if (warp == kTmaWarp) {
    // ------------------------------------------------------------------ TMA producer
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    int ahead = 0;     // k-blocks of the first unit whose weights are on their way already
    if constexpr (!GROUPED) {
      if (p.prefetch_w && blockIdx.x < num_vtiles) {
        const Work w = decode_work(blockIdx.x, p, nkb, GROUPED);
        const TileInfo t = get_tile<GROUPED>(w.tile, p, m_blocks, n_blocks, tile_m_start);
        ahead = min(kStages, w.kb_end - w.kb_begin);
        if (elect_one()) {
          for (int i = 0; i < ahead; ++i) {
            const uint32_t bar = full_bar + 8 * i;
            sa::expect_tx(bar, kABytes + t.halves * kBHalfBytes);
            for (int h = 0; h < t.halves; ++h)
              sa::tma_load_2d(smem_b + i * kBBytes + h * kBHalfBytes, &map_b, bar, (w.kb_begin + i) * BLOCK_K, t.b_row0 + h * 128);
          }
        }
        __syncwarp();
      }
      pdl_wait();
      pdl_release<kReleaseThreads>();
    }
    pdl_trigger_if(num_vtiles <= static_cast<int>(gridDim.x));
    for (int vt = blockIdx.x; ok && vt < num_vtiles; vt += gridDim.x) {
      const Work w = decode_work(vt, p, nkb, GROUPED);
      const TileInfo t = get_tile<GROUPED>(w.tile, p, m_blocks, n_blocks, tile_m_start);
      const uint32_t bytes = kABytes + t.halves * kBHalfBytes;
      for (int kb = w.kb_begin; kb < w.kb_end; ++kb) {
        if (ahead == 0) {
          ok = sa::wait(done_bar + 8 * stage, phase ^ 1u, p.status, 1);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        if (elect_one()) {
          const uint32_t bar = full_bar + 8 * stage;
          if (ahead == 0) {
            sa::expect_tx(bar, bytes);
            sa::tma_load_2d(smem_b + stage * kBBytes, &map_b, bar, kb * BLOCK_K, t.b_row0);
            if (t.halves == 2)
              sa::tma_load_2d(smem_b + stage * kBBytes + kBHalfBytes, &map_b, bar, kb * BLOCK_K, t.b_row0 + 128);
          }
          sa::tma_load_2d(smem_a + stage * kABytes, &map_a, bar, kb * BLOCK_K, t.row0);
        }
        __syncwarp();
        if (ahead > 0) --ahead;
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == kMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer
    // The whole warp walks the loop so that addresses and descriptors stay warp-uniform; one elected lane issues.
    if constexpr (!GROUPED) pdl_await_release<kReleaseThreads>();
    const uint64_t a_desc0 = umma_desc_k128(smem_a);
    const uint64_t b_desc0 = umma_desc_k128(smem_b);
    int stage = 0;
    uint32_t phase = 0, use = 0;      // k-blocks issued so far: accumulator = use & 1, parity = use >> 1 & 1
    bool ok = true;
    for (int vt = blockIdx.x; ok && vt < num_vtiles; vt += gridDim.x) {
      const Work w = decode_work(vt, p, nkb, GROUPED);
      const int halves = get_tile<GROUPED>(w.tile, p, m_blocks, n_blocks, tile_m_start).halves;
      const uint32_t idesc = umma_idesc_e4m3(TILE_M, 128 * halves);
      for (int kb = w.kb_begin; kb < w.kb_end; ++kb) {
        const int buf = static_cast<int>(use & 1u);
        ok = sa::wait(full_bar + 8 * stage, phase, p.status, 3);
        if (ok) ok = sa::wait(acc_empty + 8 * buf, ((use >> 1) & 1u) ^ 1u, p.status, 2);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        ++use;
        tc_fence_after();
        const uint64_t a_desc = a_desc0 + static_cast<uint64_t>(stage * (kABytes >> 4));
        const uint64_t b_desc = b_desc0 + static_cast<uint64_t>(stage * (kBBytes >> 4));
        if (elect_one()) {
#pragma unroll
          for (int k = 0; k < BLOCK_K / 32; ++k) {
            // advance 32 bytes along K inside the 128-byte swizzle row: +2 in the (addr >> 4) field
            umma_f8(tmem_base + static_cast<uint32_t>(buf * 256), a_desc + static_cast<uint64_t>(2 * k),
                    b_desc + static_cast<uint64_t>(2 * k), idesc, k > 0 ? 1u : 0u);
          }
          sa::commit(done_bar + 8 * stage);     // stage reusable and partial sums readable once these MMAs finish
        }
        __syncwarp();
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
  } else if (warp == kStagerWarp) {
    // ------------------------------------------------------------------ scale stager
    if constexpr (!GROUPED) pdl_wait();
    int slot = 0;
    uint32_t sphase = 0;
    bool ok = true;
    // Row-major fp32 scales whose rows start on 16 bytes: a row's four k-blocks are one 16-byte copy.
    const bool row_vec = !p.sa_ue8m0 && p.sa_stride_g == 1 && (p.sa_stride_m & 3) == 0 &&
                         (reinterpret_cast<uintptr_t>(p.sa) & 15u) == 0 && p.sa_stride_m >= ((nkb + 3) & ~3);
    for (int vt = blockIdx.x; ok && vt < num_vtiles; vt += gridDim.x) {
      const Work w = decode_work(vt, p, nkb, GROUPED);
      const TileInfo t = get_tile<GROUPED>(w.tile, p, m_blocks, n_blocks, tile_m_start);
      const float* sb_base = p.sb + static_cast<int64_t>(t.expert) * p.sb_stride_e;
      const bool vec = row_vec && (w.kb_begin & 3) == 0;
      for (int kb0 = w.kb_begin; kb0 < w.kb_end; kb0 += kScaleGroup) {
        ok = __all_sync(0xffffffffu, sa::wait(scale_empty + 8 * slot, sphase ^ 1u, p.status, 5));
        if (!ok) break;
        const uint32_t dst = smem_scale + slot * (kSlotFloats * 4);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const int rr = r * 32 + lane;
          const bool in = rr < t.valid_rows;
          const float* row = p.sa + (in ? static_cast<int64_t>(t.row0 + rr) * p.sa_stride_m : 0);
          if (p.sa_ue8m0) {
            // packed exponent bytes of four k-blocks (a unit starts on a word: the host rounds kb_per_split)
            sa::cp_async4(dst + rr * 16, row + (in ? static_cast<int64_t>(kb0 >> 2) * p.sa_stride_g : 0), in);
          } else if (vec) {
            sa::cp_async16(dst + rr * 16, row + (in ? kb0 : 0), in);
          } else {
#pragma unroll
            for (int j = 0; j < kScaleGroup; ++j) {
              const bool jn = in && kb0 + j < w.kb_end;
              sa::cp_async4(dst + rr * 16 + j * 4, row + (jn ? static_cast<int64_t>(kb0 + j) * p.sa_stride_g : 0), jn);
            }
          }
        }
        if (lane < 2 * kScaleGroup) {
          const int h = lane >> 2, kb = kb0 + (lane & 3);
          const bool in = kb < w.kb_end;
          const int nb = min(t.n0 + h * 128, p.N - 1) / 128;
          sa::cp_async4(dst + (TILE_M * kScaleGroup + lane) * 4,
                    sb_base + (in ? static_cast<int64_t>(nb) * p.sb_stride_n + static_cast<int64_t>(kb) * p.sb_stride_g : 0), in);
        }
        sa::cp_async_arrive(scale_full + 8 * slot);
        if (++slot == kScaleSlots) { slot = 0; sphase ^= 1u; }
      }
    }
    // the copies must have landed before shared memory goes away
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
  }
  } else {
    // ====================================================================== promotion + epilogue warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpiRegs));
    if constexpr (!GROUPED) pdl_await_release<kReleaseThreads>();
    // What the loop below needs is worked out again from the parameter block and the special registers: values computed
    // before the branch stay live next to 128 accumulators, and ptxas then spills (to a local memory with almost no L1).
    int m_blocks, n_blocks, nkb, num_vtiles, split_k, warp, lane;
    uint32_t tmem_base;
    {
      int tid, M = p.M, N = p.N, K = p.K;
      asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid), "+r"(M), "+r"(N), "+r"(K));
      warp = tid >> 5;
      lane = tid & 31;
      m_blocks = (M + TILE_M - 1) / TILE_M;
      n_blocks = (N + p.tile_n - 1) / p.tile_n;
      nkb = (K + BLOCK_K - 1) / BLOCK_K;
      split_k = GROUPED ? 1 : p.split_k;
      const int num_tiles = GROUPED ? tile_m_start[p.num_experts] * n_blocks : m_blocks * n_blocks;
      const int tail_first = (GROUPED || split_k == 1) ? num_tiles : p.tail_first;
      num_vtiles = tail_first + (num_tiles - tail_first) * split_k;
      tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot);
    }
    const int quad = warp & 3;         // tensor-memory lane quadrant this warp may read
    const int part = warp >> 2;        // which half of the tile's columns
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t sc_row = smem_scale + (quad * 32 + lane) * 16, sc_col = smem_scale + TILE_M * 16;
    int slot = 0, stage = 0, buf = 0;
    uint32_t phase = 0, sphase = 0;
    bool ok = true;
    for (int vt = blockIdx.x; ok && vt < num_vtiles; vt += gridDim.x) {
      int kb_begin, kb_end;
      bool wide;      // 256 columns: the warp takes 128 of them; else 64
      {
        const Work w = decode_work(vt, p, nkb, GROUPED);
        kb_begin = w.kb_begin;
        kb_end = w.kb_end;
        wide = get_tile<GROUPED>(w.tile, p, m_blocks, n_blocks, tile_m_start).halves == 2;
      }
      const int col0 = wide ? part * 128 : part * 64;
      const uint32_t sc_b = sc_col + (wide ? part * (kScaleGroup * 4) : 0);
      float acc[CPW];
#pragma unroll
      for (int c = 0; c < CPW; ++c) acc[c] = 0.f;
      // One k-block per iteration and one way out of the loop (unrolled over a scale slot's four k-blocks, with an exit in
      // each, the accumulators' copies between the paths spilled).  A k-block's scale product is fetched under the
      // read-out before it: fetched where it is needed, its latency cost 115 cycles per k-block.
      ok = sa::wait(scale_full + 8 * slot, sphase, p.status, 6);
      if (!ok) break;
      float sa_v = sa::ld_f32(sc_row + slot * (kSlotFloats * 4)), sb_v = sa::ld_f32(sc_b + slot * (kSlotFloats * 4));
#pragma unroll 1
      for (int kb = kb_begin; kb < kb_end; ++kb) {
        const int j = (kb - kb_begin) & (kScaleGroup - 1);
        if (p.sa_ue8m0) sa_v = __uint_as_float(((__float_as_uint(sa_v) >> (8 * j)) & 0xffu) << 23);   // 2 ** (byte - 127)
        const float s = sa_v * sb_v;
        const float2 s2 = make_float2(s, s);
        ok = sa::wait(done_bar + 8 * stage, phase, p.status, 4);
        if (j == kScaleGroup - 1 || kb + 1 == kb_end) {
          __syncwarp();
          sa::arrive_if(scale_empty + 8 * slot, lane == 0);      // the slot's last product is in registers
          if (++slot == kScaleSlots) { slot = 0; sphase ^= 1u; }
          if (ok && kb + 1 < kb_end) ok = sa::wait(scale_full + 8 * slot, sphase, p.status, 6);
        }
        if (!ok) break;
        tc_fence_after();
        const uint32_t taddr = tmem_base + lane_addr + static_cast<uint32_t>(buf * 256 + col0);
        const uint32_t sc_next = slot * (kSlotFloats * 4), jn = 4 * ((j + 1) & (kScaleGroup - 1));
#pragma unroll
        for (int ch = 0; ch < CPW; ch += kChunk) {
          if (ch == 64 && !wide) break;
          float v[kChunk];
          tmem_ld32(taddr + ch, v);
          tmem_ld32(taddr + ch + 32, v + 32);
          if (ch == 0) {
            sa_v = sa::ld_f32(sc_row + sc_next + (p.sa_ue8m0 ? 0 : jn));
            sb_v = sa::ld_f32(sc_b + sc_next + jn);
          }
          tmem_ld_wait();
          if (ch + kChunk == CPW || (ch + kChunk == 64 && !wide)) {
            // all of this warp's reads of the buffer are complete: hand it back to the MMA warp
            tc_fence_before();
            __syncwarp();
            sa::arrive_if(acc_empty + 8 * buf, lane == 0);
          }
          // two fp32 FMAs per instruction (fma.rn.f32x2)
#pragma unroll
          for (int c = 0; c < kChunk; c += 2) {
            const float2 r = __ffma2_rn(make_float2(v[c], v[c + 1]), s2, make_float2(acc[ch + c], acc[ch + c + 1]));
            acc[ch + c] = r.x;
            acc[ch + c + 1] = r.y;
          }
        }
        buf ^= 1;
        if (++stage == kStages) { stage = 0; phase ^= 1u; }
      }
      const Work w = decode_work(vt, p, nkb, GROUPED);
      const TileInfo t = get_tile<GROUPED>(w.tile, p, m_blocks, n_blocks, tile_m_start);
      const int row_in_tile = quad * 32 + lane;
      const int m = t.row0 + row_in_tile;
      const int n0 = t.n0 + col0;
      const int cols = min(p.N - n0, wide ? 128 : 64);
      if (ok && row_in_tile < t.valid_rows) {
        if (w.partial) {
          // partial sums: planes of whole tiles, [(tile - tail_first) * split_k + split][128][tile_n], or of the output
          float* dst = p.partial_tiles
                           ? p.partial + ((static_cast<int64_t>(w.tile - p.tail_first) * split_k + w.split) * TILE_M + row_in_tile) * p.tile_n + col0
                           : p.partial + (static_cast<int64_t>(w.split) * p.M + m) * p.N + n0;
          const bool vec_ok = p.partial_tiles || (p.N % 4) == 0;
#pragma unroll
          for (int c = 0; c < CPW; c += 16)
            if (c < cols) store_row<16>(dst + c, reinterpret_cast<const float(&)[16]>(acc[c]), cols - c, vec_ok);
        } else {
          store_out<CPW>(static_cast<OutT*>(p.out), static_cast<const OutT*>(p.bias), m, n0, p.ldo, acc, cols);
        }
      }
    }
    tc_fence_before();
    __syncthreads();
    return;
  }

  // ---------------------------------------------------------------------- common exit
  tc_fence_before();
  __syncthreads();
  if (*reinterpret_cast<volatile int*>(p.status) != 0) {
    // a wait gave up: let copies that may still be in flight land before shared memory is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// Sum of the split-K partial results, added in split order (so the result does not depend on which
// CTA finished first), converted to the output type.  One thread per four consecutive columns.
template <typename OutT>
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float* __restrict__ partial, OutT* __restrict__ out,
                                                            const OutT* __restrict__ bias, int M, int N, int64_t ldo,
                                                            int split_k) {
  pdl_start();
  const int n4 = N >> 2;
  const int64_t total = static_cast<int64_t>(M) * n4;
  const int64_t plane = static_cast<int64_t>(M) * N;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int m = static_cast<int>(i / n4), c = static_cast<int>(i % n4) * 4;
    const float* src = partial + static_cast<int64_t>(m) * N + c;
    float4 acc = __ldcs(reinterpret_cast<const float4*>(src));
    for (int s = 1; s < split_k; ++s) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(src + s * plane));
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    OutT* dst = out + static_cast<int64_t>(m) * ldo + c;
    const float vals[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      OutT v = cvt1(dst, vals[j]);
      if (bias) v = cvt1(dst, static_cast<float>(v) + static_cast<float>(bias[c + j]));
      dst[j] = v;
    }
  }
}

template <typename OutT>
int launch_reduce(const GemmParams& p, cudaStream_t stream) {
  const int64_t total = static_cast<int64_t>(p.M) * (p.N >> 2);
  int64_t blocks = (total + 255) / 256;
  if (blocks > 4 * sm_count()) blocks = 4 * sm_count();
  launch_pdl(splitk_reduce_kernel<OutT>, static_cast<int>(blocks), 256, 0, stream, p.partial, static_cast<OutT*>(p.out),
             static_cast<const OutT*>(p.bias), p.M, p.N, p.ldo, p.split_k);
  B200_CUDA_TRY(cudaGetLastError());
  return B200_OK;
}

// Sum of the split tiles' partial planes, added in split order, converted and written into the output tile with its row
// / column bounds.  grid = (split tiles, 16 slices of 8 rows): a tile's planes are megabytes, so one block per tile would
// make this kernel longer than the wave it saves.
constexpr int kTailSlices = 16;
template <typename OutT>
__global__ void __launch_bounds__(256) tail_reduce_kernel(const float* __restrict__ partial, OutT* __restrict__ out,
                                                          const OutT* __restrict__ bias, int M, int N, int64_t ldo, int split_k, int tail_first,
                                                          int m_blocks, int n_blocks, int tile_n) {
  pdl_start();
  int m_blk, n_blk;
  tile_coords(tail_first + blockIdx.x, m_blocks, n_blocks, m_blk, n_blk);
  const int64_t plane = static_cast<int64_t>(TILE_M) * tile_n;
  const float* base = partial + static_cast<int64_t>(blockIdx.x) * split_k * plane;
  constexpr int kRows = TILE_M / kTailSlices;
  const int vecs = tile_n >> 2;
  for (int i = threadIdx.x; i < kRows * vecs; i += blockDim.x) {
    const int r = blockIdx.y * kRows + i / vecs, c = (i % vecs) * 4;
    const int m = m_blk * TILE_M + r, n = n_blk * tile_n + c;
    if (m >= M || n >= N) continue;
    const float* src = base + static_cast<int64_t>(r) * tile_n + c;
    float4 acc = __ldcs(reinterpret_cast<const float4*>(src));
    for (int s = 1; s < split_k; ++s) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(src + s * plane));
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    OutT* dst = out + static_cast<int64_t>(m) * ldo + n;
    const float vals[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N) {
        OutT v = cvt1(dst, vals[j]);
        if (bias) v = cvt1(dst, static_cast<float>(v) + static_cast<float>(bias[n + j]));
        dst[j] = v;
      }
  }
}

template <typename OutT>
int launch_tail_reduce(const GemmParams& p, cudaStream_t stream) {
  const int m_blocks = (p.M + TILE_M - 1) / TILE_M;
  const int n_blocks = (p.N + p.tile_n - 1) / p.tile_n;
  const dim3 grid(m_blocks * n_blocks - p.tail_first, kTailSlices);
  launch_pdl(tail_reduce_kernel<OutT>, grid, 256, 0, stream, p.partial, static_cast<OutT*>(p.out),
             static_cast<const OutT*>(p.bias), p.M, p.N, p.ldo, p.split_k, p.tail_first, m_blocks, n_blocks, p.tile_n);
  B200_CUDA_TRY(cudaGetLastError());
  return B200_OK;
}

int reduce_partials(const GemmParams& p, cudaStream_t stream) {
  switch (p.out_dtype) {
    case B200_DT_BF16: return p.partial_tiles ? launch_tail_reduce<__nv_bfloat16>(p, stream) : launch_reduce<__nv_bfloat16>(p, stream);
    case B200_DT_F16: return p.partial_tiles ? launch_tail_reduce<__half>(p, stream) : launch_reduce<__half>(p, stream);
    default: return p.partial_tiles ? launch_tail_reduce<float>(p, stream) : launch_reduce<float>(p, stream);
  }
}

// ------------------------------------------------------------------------------------ host
template <bool GROUPED, typename OutT>
int launch(const CUtensorMap& ma, const CUtensorMap& mb, const GemmParams& p, cudaStream_t stream) {
  auto kern = gemm_block_fp8_kernel<GROUPED, OutT>;
  static bool attr_set[64] = {false};
  int dev = 0;
  B200_CUDA_TRY(cudaGetDevice(&dev));
  dev &= 63;
  if (!attr_set[dev]) {
    B200_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes));
    attr_set[dev] = true;
  }
  const long long m_blocks = (p.M + TILE_M - 1) / TILE_M;
  const long long n_blocks = (p.N + p.tile_n - 1) / p.tile_n;
  // grouped: the tile count lives on the device; row tiles <= ceil(rows/128) + experts bounds the grid
  const long long dense_tiles = m_blocks * n_blocks;
  const long long split_from = p.split_k == 1 ? dense_tiles : p.tail_first;
  const long long tiles = GROUPED ? (m_blocks + p.num_experts) * n_blocks
                                  : split_from + (dense_tiles - split_from) * p.split_k;
  if (tiles > 0x7fffffffLL) return B200_ERR_TOO_LARGE;   // the kernels count tiles in 32 bits
  const int grid = tiles < sm_count() ? static_cast<int>(tiles) : sm_count();
  B200_CUDA_TRY(launch_overlap(tiles <= sm_count(), kern, dim3(grid), dim3(kThreads), kSmemBytes, stream, ma, mb, p));
  return B200_OK;
}

template <bool GROUPED>
int launch_dtype(const CUtensorMap& ma, const CUtensorMap& mb, const GemmParams& p, cudaStream_t stream) {
  switch (p.out_dtype) {
    case B200_DT_BF16: return launch<GROUPED, __nv_bfloat16>(ma, mb, p, stream);
    case B200_DT_F16: return launch<GROUPED, __half>(ma, mb, p, stream);
    case B200_DT_F32: return launch<GROUPED, float>(ma, mb, p, stream);
    default: return B200_ERR_BAD_DTYPE;
  }
}

}  // namespace

// Kernel override for the tests, so that every kernel is reached on every shape: 0 = automatic,
// 128 / 256 = this file's kernel with that tile width, 3 / 3032 / 3064 / 3128 and 4: see below.
int g_force_block_n = 0;

int launch_gemm_swapab(const void* a, int64_t lda, int64_t a_rows, const void* b, int64_t ldb, int64_t w_rows,
                       const GemmParams& p, bool grouped, int token_tile, cudaStream_t stream);

// g_force_block_n values that select the weight-streaming (swapped-operand) kernel: 3 = token tile
// chosen from the shape, 3032 / 3064 / 3128 = that token tile; 4 = never use it.
inline int forced_token_tile() {
  return g_force_block_n == 3032 ? 32 : g_force_block_n == 3064 ? 64 : g_force_block_n == 3128 ? 128 : 0;
}

namespace {

// Which kernel a dense problem gets.  Up to 64 tokens the weight-streaming kernel (gemm_swapab.cu, 128 weight rows x up to
// 64 tokens per tile): 0-30 % faster than this file's tiles on every projection.  For 65-192 tokens it has two or three
// token tiles per weight tile, the second and third reading the weights from L2, and stays ahead (0-25 %) only while all
// of them run at once; in several waves it re-reads more than it saves.  128 tokens, us, weight-streaming / this file's:
// [4096, 7168] 14.2 / 16.8 (64 tiles), [8192, 8192] 21.0 / 26.6 (128), [10240, 8192] 35.2 / 28.4 (160),
// [36864, 7168] 62.1 / 49.6 (576); 192 tokens: [5120, 8192] 19.1 / 29.1 (120), [7168, 9216] 35.9 / 30.7 (168).  With
// three token tiles two well-filled waves still pass ([10240, 8192], 240 tiles: 33.4 / 35.1).
constexpr int64_t kStreamTokens = 192;
inline int dense_token_tile(int64_t M) { return M <= 32 ? 32 : 64; }
inline bool dense_uses_swapab(int64_t M, int64_t N, int sms) {
  if (M <= 64 || M > kStreamTokens) return M <= 64;
  const int64_t tiles = ((M + 63) / 64) * ((N + 127) / 128);
  return tiles <= sms || (M > 128 && 2 * tiles > 3 * sms && tiles <= 2 * sms);
}

// Split count of the weight-streaming kernel: when the output has too few tiles for the SMs, the k-blocks of each tile are
// spread over several CTAs so that the weights stream through all SMs at once.
int plan_split_k(int64_t M, int64_t N, int64_t K, int sms) {
  if ((N % 4) != 0) return 1;
  const int64_t tt = dense_token_tile(M);
  const int64_t tiles = ((M + tt - 1) / tt) * ((N + 127) / 128);
  const int64_t nkb = (K + BLOCK_K - 1) / BLOCK_K;
  // measured on DeepSeek-V3 shapes: below 32 k-blocks the launch and pipeline ramp dominate and the
  // extra reduce kernel costs more than the idle SMs
  if (nkb < 32) return 1;
  if (tiles * 2 > sms) {
    // More tiles than half the SMs: split only to fill a last wave that is mostly empty.
    auto fill = [sms](int64_t t) { return static_cast<double>(t) / static_cast<double>(((t + sms - 1) / sms) * sms); };
    if (fill(tiles) >= 0.7) return 1;
    for (int s2 = 2; s2 <= 4; ++s2)
      if (nkb / s2 >= 8 && fill(tiles * s2) >= 0.75) return s2;
    return 1;
  }
  // (A byte model that picks the count with the best fill of the SMs' wave slots -- 5 for 56 tiles, 3 for 80 -- was
  // measured no better than this rule: 31.5 against 30.1 us on the 56-tile down projection at 64 tokens, 23.8 against
  // 22.5 us on the 80-tile qkv projection; fewer CTAs each pull more than their share of the HBM bandwidth.)
  int64_t s = sms / tiles;
  if (s > nkb / 8) s = nkb / 8;  // at least eight k-blocks per CTA
  if (s > 16) s = 16;
  return s < 2 ? 1 : static_cast<int>(s);
}

// Split-K workspace: split_k fp32 planes of [M, N].  (Folding the sum into the GEMM kernel -- the CTA that
// completes a tile's last split adds the planes -- was measured slower than the second kernel at every M:
// the device-wide fences and the CTA-wide meeting it needs cost more than a launch.)
inline size_t splitk_workspace_bytes(int split_k, int64_t M, int64_t N) {
  return static_cast<size_t>(split_k) * M * N * sizeof(float);
}

// Schedule of this file's kernel for a dense problem: tile width, and how many of the last tiles have their k-blocks
// divided among several CTAs.  A CTA works through the tiles with a fixed stride, so a last wave that fills few of the
// SMs costs as much as a full one, and a problem of fewer tiles than SMs leaves the rest idle: the k-blocks of just
// those tiles are spread over the idle SMs, each writing fp32 planes that a second kernel adds in split order.
// Cost in cycles of the longest CTA: its k-blocks at the measured rate of the tile width (a 128-column k-block costs nearly
// as much as a 256-column one: the read-out's waits and the way round the pipeline are the same), a tile's ramp and
// epilogue, and for a split the second kernel (about 5 us) and the planes' round trip through L2 (about 3 TB/s).
struct TilePlan {
  int tile_n = 256, split_k = 1, kb_per_split = 0, tail_first = 0;
  size_t bytes = 0;
};
TilePlan plan_tiles(int64_t M, int64_t N, int64_t K, int sms, size_t max_bytes) {
  const int64_t nkb = (K + BLOCK_K - 1) / BLOCK_K;
  TilePlan best;
  double best_cost = 0;
  for (const int tile_n : {256, 128}) {
    const double kb_cycles = tile_n == 256 ? 850.0 : 720.0, tile_cycles = 2500.0;
    const int64_t tiles = ((M + TILE_M - 1) / TILE_M) * ((N + tile_n - 1) / tile_n);
    const int64_t full = tiles / sms, rest = tiles % sms;
    auto consider = [&](const TilePlan& q, double cost) {
      if (best_cost == 0 || cost < best_cost) { best = q; best_cost = cost; }
    };
    TilePlan q;
    q.tile_n = tile_n;
    const double wave = nkb * kb_cycles + tile_cycles;
    consider(q, static_cast<double>(full + (rest ? 1 : 0)) * wave);
    // below 32 k-blocks (16 when only a tail is split) the second kernel costs more than the idle SMs
    if (rest == 0 || tiles > 0x3fffffff || nkb < (full ? 16 : 32)) continue;
    const int64_t most = std::min<int64_t>({sms / rest, nkb / 4, 32});
    for (int64_t s = 2; s <= most; ++s) {
      q.kb_per_split = static_cast<int>((nkb + s - 1) / s);
      q.split_k = static_cast<int>((nkb + q.kb_per_split - 1) / q.kb_per_split);
      q.tail_first = static_cast<int>(tiles - rest);
      q.bytes = static_cast<size_t>(rest) * q.split_k * TILE_M * tile_n * sizeof(float);
      if (q.split_k < 2 || q.bytes > max_bytes) continue;
      consider(q, static_cast<double>(full) * wave + q.kb_per_split * kb_cycles + tile_cycles + 9000.0 + 2.0 * q.bytes / 1700.0);
    }
  }
  return best;
}

// What a dense problem runs with a workspace of up to max_bytes: the one answer behind dense_mm, the plan and the
// workspace entry points.  bytes = workspace the schedule uses, 0 when nothing is split.
struct DensePlan {
  bool swapab = false;
  int split_k = 1;        // CTAs per divided tile, either kernel
  size_t bytes = 0;
  TilePlan tiles;         // this file's kernel
};
DensePlan plan_dense(int64_t M, int64_t N, int64_t K, int sms, bool swapab, size_t max_bytes) {
  DensePlan d;
  d.swapab = swapab;
  if (swapab) {
    const int s = plan_split_k(M, N, K, sms);
    const size_t bytes = s > 1 ? splitk_workspace_bytes(s, M, N) : 0;
    if (bytes <= max_bytes) {
      d.split_k = s;
      d.bytes = bytes;
    }
  } else {
    d.tiles = plan_tiles(M, N, K, sms, max_bytes);
    d.split_k = d.tiles.split_k;
    d.bytes = d.tiles.bytes;
  }
  return d;
}

}  // namespace

// A linear with power-of-two scales on both operands: whether the promoting kernels of this file and gemm_swapab.cu take the
// product (exponent bytes decoded to fp32 scales) instead of the block-scaling one, which accumulates in tensor memory
// without read-outs but cannot divide a tile's k-blocks.  us with the quantiser, promoting / block-scaling:
//   few tiles: 16 x 7168 x 18432 28 / 49, 128 x 8192 x 8192 22 / 27, 256 x 1280 x 8192 18 / 26
//   up to 64 rows: 64 x 10240 x 8192 25.4 / 27.3, 64 x 18432 x 7168 28.3 / 30.3
//   its 128 x 128 tiles fill more than half of the SMs once: below K = 16384 the two are within 6 % of each other
//     (128 x 10240 x 12288 42.0 / 39.3, 256 x 8192 x 14336 48.8 / 46.8, 256 x 7168 x 8192 28.3 / 29.1) but for nearly full
//     waves, whose tiles leave no SMs to divide k-blocks over (128 x 18432 x 14336 66 / 54); above it the splits lead
//     (512 x 4096 x 16384 50.8 / 52.5, 256 x 7168 x 18432 54.6 / 56.5, 128 x 10240 x 28672 71 / 83), again but for nearly
//     full waves, where this rule gives 7-15 % away (128 x 18432 x 16384 72 / 63, x 28672 107 / 100)
//   more than one such wave: 640 x 57344 x 8192 281 / 317, 768 x 7168 x 18432 105 / 150, 320 x 36864 x 7168 96 / 103;
//     on wide outputs the lead is gone by 768 rows (768 x 36864 x 7168 185 / 183, 1023 x 36864 x 7168 243 / 237)
//   from 1024 rows on: 1024 x 7168 x 18432 141 / 128, 2048 x 8192 x 8192 135 / 131
bool packed_promotes(int64_t M, int64_t N, int64_t K) {
  const int64_t tiles = ((M + 127) / 128) * ((N + 127) / 128);
  const bool one_full_wave = tiles <= sm_count() && 2 * tiles > sm_count();
  return M < 1024 && !(one_full_wave && M > 64 && K < 16384);
}

int dense_mm(const void* a, int64_t lda, const void* b, int64_t ldb, const float* sa, int64_t sa_stride_m,
             int64_t sa_stride_g, const float* sb, int64_t sb_stride_n, int64_t sb_stride_g, void* out, int64_t ldo,
             int out_dtype, int64_t M, int64_t N, int64_t K, int split_k, void* workspace, size_t workspace_bytes,
             void* stream, int sa_ue8m0, const void* bias, int prefetch_w) {
  if (M < 0 || N < 0 || K <= 0) return B200_ERR_BAD_SHAPE;
  if (M == 0 || N == 0) return B200_OK;
  if (M > 0x7fffff00LL || N > 0x7fffff00LL || K > 0x7fffff00LL) return B200_ERR_TOO_LARGE;
  if (!a || !b || !sa || !sb || !out) return B200_ERR_NULL_PTR;
  if (out_dtype != B200_DT_BF16 && out_dtype != B200_DT_F16 && out_dtype != B200_DT_F32) return B200_ERR_BAD_DTYPE;
  if (lda < K || ldb < K || ldo < N) return B200_ERR_BAD_STRIDE;
  if ((lda % 16) != 0 || (ldb % 16) != 0 || !aligned16(a) || !aligned16(b)) return B200_ERR_MISALIGNED;
  if (sa_stride_m < 0 || sa_stride_g < 0 || sb_stride_n < 0 || sb_stride_g < 0) return B200_ERR_BAD_STRIDE;
  const int nkb = static_cast<int>((K + BLOCK_K - 1) / BLOCK_K);
  if (split_k < 0 || split_k > 64) return B200_ERR_BAD_SHAPE;
  if (split_k > 1) {
    if ((N % 4) != 0 || split_k > nkb) return B200_ERR_BAD_SHAPE;
    if (!workspace) return B200_ERR_NULL_PTR;
    if (!aligned16(workspace)) return B200_ERR_MISALIGNED;
    if (workspace_bytes < splitk_workspace_bytes(split_k, M, N)) return B200_ERR_TOO_LARGE;
  }
  int rc = require_sm100();
  if (rc != B200_OK) return rc;
  if (gemm_sticky_status() != 0) return B200_ERR_DEVICE_TIMEOUT;   // sticky until b200_gemm_device_status clears it
  TilePlan plan;
  const bool swapab = g_force_block_n == 3 || forced_token_tile() != 0 || (g_force_block_n == 0 && dense_uses_swapab(M, N, sm_count()));
  if (split_k <= 1) {
    // automatic (0): split only when the caller gave room for it
    const size_t room = split_k == 0 && workspace && aligned16(workspace) ? workspace_bytes : 0;
    const DensePlan d = plan_dense(M, N, K, sm_count(), swapab, room);
    plan = d.tiles;
    split_k = swapab ? d.split_k : 1;
  }
  if (g_force_block_n == 128 || g_force_block_n == 256) {
    plan = TilePlan();
    plan.tile_n = g_force_block_n;
  }

  GemmParams p;
  p.sa = sa; p.sb = sb; p.out = out;
  p.sa_stride_m = sa_stride_m; p.sa_stride_g = sa_stride_g;
  p.sb_stride_n = sb_stride_n; p.sb_stride_g = sb_stride_g;
  p.ldo = ldo;
  p.M = static_cast<int>(M); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
  p.out_dtype = out_dtype;
  p.status = gemm_status_ptr();
  p.expert_offsets = nullptr; p.problem_sizes = nullptr; p.sb_stride_e = 0; p.num_experts = 0;
  p.split_k = split_k < 1 ? 1 : split_k;
  p.kb_per_split = (nkb + p.split_k - 1) / p.split_k;
  // every split must own at least one k-block (an empty one would store zeros, which is still right,
  // but the count is trimmed so that no CTA is launched for nothing)
  p.split_k = (nkb + p.kb_per_split - 1) / p.kb_per_split;
  p.tail_first = 0;
  p.partial_tiles = 0;
  p.bias = bias;
  p.prefetch_w = prefetch_w;
  p.tile_n = plan.tile_n;
  if (plan.split_k > 1) {
    p.split_k = plan.split_k;
    p.kb_per_split = plan.kb_per_split;
    p.tail_first = plan.tail_first;
    p.partial_tiles = 1;
  }
  if (sa_ue8m0 && p.split_k > 1 && (p.kb_per_split & 3) != 0) {
    p.kb_per_split = (p.kb_per_split + 3) & ~3;     // a unit starts on a packed exponent word
    p.split_k = (nkb + p.kb_per_split - 1) / p.kb_per_split;
  }
  p.partial = static_cast<float*>(workspace);
  p.sa_ue8m0 = sa_ue8m0;
  if (!p.status) return B200_ERR_CUDA;

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (swapab) {
    int tt = forced_token_tile();
    if (tt == 0) tt = dense_token_tile(M);
    rc = launch_gemm_swapab(a, lda, M, b, ldb, N, p, false, tt, st);
  } else {
    CUtensorMap ma, mb;
    rc = make_map_u8_2d(&ma, a, M, K, lda, TILE_M);
    if (rc != B200_OK) return rc;
    rc = make_map_u8_2d(&mb, b, N, K, ldb, 128);
    if (rc != B200_OK) return rc;
    rc = launch_dtype<false>(ma, mb, p, st);
  }
  if (rc != B200_OK || p.split_k == 1) return rc;
  return reduce_partials(p, st);
}

}  // namespace b200

extern "C" int b200_fp8_blockwise_scaled_mm(const void* a, int64_t lda, const void* b, int64_t ldb, const float* sa,
                                            int64_t sa_stride_m, int64_t sa_stride_g, const float* sb,
                                            int64_t sb_stride_n, int64_t sb_stride_g, void* out, int64_t ldo,
                                            int out_dtype, int64_t M, int64_t N, int64_t K, void* stream) {
  return b200::dense_mm(a, lda, b, ldb, sa, sa_stride_m, sa_stride_g, sb, sb_stride_n, sb_stride_g, out, ldo, out_dtype,
                        M, N, K, 1, nullptr, 0, stream, 0, nullptr, 0);
}

extern "C" int b200_fp8_blockwise_scaled_mm_splitk(const void* a, int64_t lda, const void* b, int64_t ldb,
                                                   const float* sa, int64_t sa_stride_m, int64_t sa_stride_g,
                                                   const float* sb, int64_t sb_stride_n, int64_t sb_stride_g, void* out,
                                                   int64_t ldo, int out_dtype, int64_t M, int64_t N, int64_t K,
                                                   int split_k, void* workspace, size_t workspace_bytes, void* stream) {
  return b200::dense_mm(a, lda, b, ldb, sa, sa_stride_m, sa_stride_g, sb, sb_stride_n, sb_stride_g, out, ldo, out_dtype,
                        M, N, K, split_k, workspace, workspace_bytes, stream, 0, nullptr, 0);
}

extern "C" int b200_fp8_blockwise_scaled_mm_ue8m0(const void* a, int64_t lda, const void* b, int64_t ldb,
                                                  const uint32_t* sa_packed, int64_t sa_stride_m, int64_t sa_stride_pack,
                                                  const float* sb, int64_t sb_stride_n, int64_t sb_stride_g, void* out,
                                                  int64_t ldo, int out_dtype, int64_t M, int64_t N, int64_t K,
                                                  void* stream) {
  return b200::dense_mm(a, lda, b, ldb, reinterpret_cast<const float*>(sa_packed), sa_stride_m, sa_stride_pack, sb,
                        sb_stride_n, sb_stride_g, out, ldo, out_dtype, M, N, K, 1, nullptr, 0, stream, 1, nullptr, 0);
}

extern "C" int b200_fp8_blockwise_scaled_mm_splitk_plan(int64_t M, int64_t N, int64_t K, int sm_count, int* split_k,
                                                        size_t* workspace_bytes) {
  if (M < 0 || N < 0 || K <= 0) return B200_ERR_BAD_SHAPE;
  if (!split_k || !workspace_bytes) return B200_ERR_NULL_PTR;
  const int sms = sm_count > 0 ? sm_count : 148;
  *split_k = 1;
  *workspace_bytes = 0;
  if (M == 0 || N == 0) return B200_OK;
  const b200::DensePlan d = b200::plan_dense(M, N, K, sms, b200::dense_uses_swapab(M, N, sms), ~size_t(0));
  *split_k = d.split_k;
  *workspace_bytes = d.bytes;
  return B200_OK;
}

extern "C" int b200_fp8_blockwise_scaled_grouped_mm(const void* a, int64_t lda, const void* b, int64_t ldb,
                                                    const float* sa, int64_t sa_stride_m, int64_t sa_stride_g,
                                                    const float* sb, int64_t sb_stride_e, int64_t sb_stride_n,
                                                    int64_t sb_stride_g, void* out, int64_t ldo, int out_dtype,
                                                    const int32_t* expert_offsets, const int32_t* problem_sizes,
                                                    int num_experts, int64_t total_rows, int64_t N, int64_t K,
                                                    void* stream) {
  using namespace b200;
  if (total_rows < 0 || N < 0 || K <= 0 || num_experts <= 0) return B200_ERR_BAD_SHAPE;
  if (total_rows == 0 || N == 0) return B200_OK;
  if (num_experts > kMaxExperts) return B200_ERR_TOO_LARGE;
  if (total_rows > 0x7fffff00LL || K > 0x7fffff00LL || N * num_experts > 0x7fffff00LL) return B200_ERR_TOO_LARGE;
  if (!a || !b || !sa || !sb || !out || !expert_offsets || !problem_sizes) return B200_ERR_NULL_PTR;
  if (out_dtype != B200_DT_BF16 && out_dtype != B200_DT_F16 && out_dtype != B200_DT_F32) return B200_ERR_BAD_DTYPE;
  if (lda < K || ldb < K || ldo < N) return B200_ERR_BAD_STRIDE;
  if ((lda % 16) != 0 || (ldb % 16) != 0 || !aligned16(a) || !aligned16(b)) return B200_ERR_MISALIGNED;
  if (sa_stride_m < 0 || sa_stride_g < 0 || sb_stride_e < 0 || sb_stride_n < 0 || sb_stride_g < 0)
    return B200_ERR_BAD_STRIDE;
  // an expert's weights are rows [e*N, (e+1)*N) of one matrix and its scales are indexed by 128-row block:
  // with N % 128 != 0 both would straddle experts
  if (N % 128 != 0) return B200_ERR_BAD_SHAPE;
  int rc = require_sm100();
  if (rc != B200_OK) return rc;
  if (gemm_sticky_status() != 0) return B200_ERR_DEVICE_TIMEOUT;

  GemmParams p;
  p.sa = sa; p.sb = sb; p.out = out;
  p.sa_stride_m = sa_stride_m; p.sa_stride_g = sa_stride_g;
  p.sb_stride_n = sb_stride_n; p.sb_stride_g = sb_stride_g; p.sb_stride_e = sb_stride_e;
  p.ldo = ldo;
  p.M = static_cast<int>(total_rows); p.N = static_cast<int>(N); p.K = static_cast<int>(K);
  p.out_dtype = out_dtype;
  p.status = gemm_status_ptr();
  p.expert_offsets = expert_offsets; p.problem_sizes = problem_sizes; p.num_experts = num_experts;
  p.split_k = 1; p.kb_per_split = 0; p.partial = nullptr; p.tail_first = 0; p.sa_ue8m0 = 0;
  p.partial_tiles = 0; p.tile_n = 256; p.bias = nullptr; p.prefetch_w = 0;
  if (!p.status) return B200_ERR_CUDA;

  // An expert's weights are rows [e*N, (e+1)*N) of one [E*N, K] matrix.
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // Up to 56 rows per expert on average the weight-streaming kernel is used: measured on 64 experts of [4096, 7168] it takes
  // 293 us against 316 at 40 rows, the same at 56 and 444 against 325 at 80.  (Two ways to spare experts of 129-190 rows
  // their second row tile were built and measured at 128 rows, 386 us: tokens on the MMA's N side, 440-500 us -- the
  // 16-lane tensor-memory loads it needs are 3.3 times slower than the 32-lane ones -- and 192-row x 128-column tiles,
  // 495 us -- half as many weight bytes in flight per hand-off.)
  const int64_t avg_rows = total_rows / num_experts;
  const bool auto_swap = g_force_block_n == 0 && avg_rows <= 56;
  if ((g_force_block_n == 3 || forced_token_tile() != 0 || auto_swap) && N % 128 == 0) {
    int tt = forced_token_tile();
    if (tt == 0) tt = avg_rows <= 20 ? 32 : 64;
    return launch_gemm_swapab(a, lda, total_rows, b, ldb, N * num_experts, p, true, tt, st);
  }
  // 256-wide tiles unless they would leave half of the SMs idle; a 128-column remainder (N % 256 != 0) costs its half only.
  const int64_t tiles = (total_rows / TILE_M + num_experts) * ((N + 255) / 256);
  p.tile_n = g_force_block_n == 128 || (g_force_block_n != 256 && 2 * tiles < sm_count()) ? 128 : 256;
  CUtensorMap ma, mb;
  rc = make_map_u8_2d(&ma, a, total_rows, K, lda, TILE_M);
  if (rc != B200_OK) return rc;
  rc = make_map_u8_2d(&mb, b, N * num_experts, K, ldb, 128);
  if (rc != B200_OK) return rc;
  return launch_dtype<true>(ma, mb, p, st);
}

extern "C" int b200_debug_force_block_n(int block_n) {
  b200::g_force_block_n = block_n;
  return B200_OK;
}

extern "C" size_t b200_fp8_blockwise_scaled_mm_workspace_bytes(int64_t M, int64_t N, int64_t K) {
  using namespace b200;
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  return plan_dense(M, N, K, sm_count(), dense_uses_swapab(M, N, sm_count()), ~size_t(0)).bytes;
}
