// W4A16 contractions with the weights as the stationary operand in tensor memory (tcgen05, A from TMEM).
//
//   Y[m, n] = T( sum_k f32(X[m, k]) * f32( T( (q[k, n] - 8) * S[k / G, n] ) ) )
//
// Program: weight_only_int4_matmul (reference kernel body examples/kernels/contraction/weight_only_int4.py:18-51)
// and the MoE grouped contractions (examples/kernels/ragged/grouped_gemm.py:11-70, ragged/moe.py:12-53 with int4
// expert weights); the same arithmetic and the same order of the k blocks as w4a16_gemm.cu.
//
// Here the product is turned round: the M index of the MMA is the weight column, its N index the activation row.
// A lane of tensor memory is one weight column, so the thread that expands a column's packed words stores them
// straight into its own lane (tcgen05.st, 64 columns of 32 bits per 128 k) and the tensor core reads them from there.
// The expanded weights never pass through shared memory, and a tile has as many rows as the call has, in steps of
// 16, instead of 128.
//
// What bounds it: per 128 k 600 cycles for a lone tile or a pair of up to 128 rows with all SMs at work - the issue loop (450 of
// them) and the dequantisers, 320 issue slots of every scheduler (290 with the scales in f32), hand their blocks to each other; with neither
// conversion nor more than one MMA a block it is 560.  At 256 rows of a pair the MMAs' 1024 cycles count.  A small call is start-up (the
// wait for the kernel ahead ends 1.3 us after that kernel, first words 1 us later), its k blocks and the exchange between
// the CTAs of a cluster (2 us).  Against the forms with the weights in shared memory: M77 K14336 N4096 81.1 -> 14.7 us,
// M1024 K4096 N4096 50.9 -> 25.3, 64 tokens on 64 experts of 4096 x 1408 414 -> 157 (the whole layer).
#include <algorithm>
#include <type_traits>

#include "cluster.cuh"
#include "common.cuh"
#include "tma.cuh"
#include "umma.cuh"
#include "w4a16_tmem.cuh"

namespace ib200 {

__device__ int g_w4a16_tmem_status = 0;

namespace {

constexpr int BK = 128;                    // k per stage
constexpr int COLS = 128;                  // weight columns of a CTA's tile (lanes of tensor memory)
constexpr int W_ROWS = BK / 8;             // packed rows of a stage
constexpr int W_BYTES = W_ROWS * COLS * 4;
constexpr int S_BYTES = 1024;              // room for the scales of a stage: up to four groups of 128 columns
constexpr int W_STAGE = W_BYTES + S_BYTES;
constexpr int SETS = 4;                    // sets of four dequantiser warps that take turns at the k blocks
constexpr int A_STAGES = SETS;             // stages of expanded weights, 64 columns of tensor memory each
constexpr int A_COLUMN = 256;              // first tensor-memory column of the expanded weights
constexpr int ACC_COLUMNS = 256;           // tensor-memory columns of the accumulators (two sets up to 128 rows)
constexpr int FIRST_EPILOGUE = 4, FIRST_DEQUANT = 8;   // multiples of four: warp % 4 is the TMEM quadrant
constexpr int THREADS = (FIRST_DEQUANT + 4 * SETS) * 32;
constexpr int LIST_BLOCKS = 1024;          // most 128-row blocks of a grouped call
constexpr int SMEM_LIMIT = 227 * 1024;

struct TmemParams {
  void* y;
  int M, K;                  // rows and width of the activations
  int WN, out_cols;          // columns of the weight matrix and of the output
  int k_blocks;              // ceil(K / 128)
  int m_tiles, n_tiles;      // row tiles; column tiles of 128 * CG weight columns
  int row_tile;              // most rows of a tile, a multiple of 16 * CG
  int box_rows;              // rows of one activation box
  int x_stages;              // stages of activations, A_STAGES .. 8
  int w_stages;              // stages of packed words, 2 * SETS .. 16
  int acc_sets;              // accumulator sets that alternate between tiles
  int split;                 // CTAs of a cluster that share a tile's k blocks (1 = none)
  int kb_each, kb_extra;     // k blocks of a CTA: the first kb_extra ranks of a cluster take one more
  uint32_t exchange;         // split: offset of the room for the cluster's partial sums, 0 = where the operands were
  uint32_t tile_magic;       // ceil(2^32 / d), d the number of tiles that vary fastest (0 stands for d = 1)
  int group_shift;           // log2 of the group size
  int twos_complement;
  // grouped modes
  const int* total_rows;     // padded row count (device)
  const int* tile_expert;    // expert of each block of `block_rows` rows
  int block_rows;
  int list_items;            // entries of the list of tiles: most items of a CTA (list_by_item), or all tiles
  int list_by_item;
  int experts;
  const int* row_route;      // route of every row; a row with no route in [0, routes) is padding; null: all rows count
  const float* route_weight; // MODE_DOWN_SCATTER: [routes]
  int routes, top_k;
  float4* clear;             // MODE_UPGATE_SILU: filled with zeros by a warp that has nothing else to do; may be null
  int64_t clear_vectors;
  int clear_pause;           // nanoseconds after each piece of 2 KiB
};

// MODE_SKINNY: dense calls of at most SKINNY_ROWS rows, as precise as the bandwidth kernels that serve the others: the
// weights go to the tensor core as the integers q - 8, exactly; every quantisation group has an accumulator of its own,
// which the epilogue warps scale and add up in f32 while the next k blocks are multiplied.
constexpr int MODE_DENSE = 0, MODE_UPGATE_SILU = 1, MODE_GROUPED_F32 = 2, MODE_DOWN_SCATTER = 3, MODE_SKINNY = 4;
constexpr int SKINNY_ROWS = 16, RING = 4;    // accumulators of RING k blocks in flight, up to four groups each
constexpr uint32_t LAST_TILE = 2;            // other modes: the barrier of tmem_full for a CTA's last tile
constexpr int GROUP_ACC = 4 * SKINNY_ROWS;   // columns of a k block's accumulators
static_assert(RING * GROUP_ACC <= ACC_COLUMNS && ACC_COLUMNS <= A_COLUMN, "accumulators end where the expanded weights begin");
static_assert(A_COLUMN + A_STAGES * 64 <= 512, "columns of tensor memory");
static_assert(LAST_TILE >= 2 && LAST_TILE < RING, "a barrier that no accumulator set has");
__host__ __device__ constexpr bool dense_mode(int mode) { return mode == MODE_DENSE || mode == MODE_SKINNY; }

// D[tmem] (+)= A[tmem] * B[smem]
template <int CG>
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                            bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  if (CG == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(acc)
        : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp writes lane (base lane + i)
__device__ __forceinline__ void tmem_store_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 16 columns
__device__ __forceinline__ void tmem_load_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
  uint16_t v;
  asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
  return v;
}

// Four neighbouring lanes hold a column each, with rows 0 and 1 in `low` and rows 2 and 3 in `high`: each gets row
// `lane & 3` of the four columns.
__device__ __forceinline__ uint2 swap_rows(uint32_t low, uint32_t high, int lane) {
  const bool odd = lane & 1, upper = lane & 2;
  const uint32_t got = __shfl_xor_sync(0xffffffffu, prmt(low, high, odd ? 0x5410 : 0x7632), 1);
  const uint32_t a = prmt(low, got, odd ? 0x3254 : 0x5410), b = prmt(high, got, odd ? 0x3276 : 0x7610);
  const uint32_t other = __shfl_xor_sync(0xffffffffu, upper ? a : b, 2);
  return upper ? make_uint2(other, b) : make_uint2(a, other);
}

template <typename T, int MODE, int CG>
__global__ void __launch_bounds__(THREADS, 1)
w4a16_tmem_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                  const __grid_constant__ CUtensorMap map_s, const TmemParams p) {
  extern __shared__ unsigned char smem_raw[];
  // Programmatic launch: a CTA of the next such launch may set itself up on an SM that this one has left, and this launch
  // touches no global memory before everything ahead of it in the stream has completed.  One call after another:
  // M16 K4096 N4096 10.3 -> 8.4 us, M77 K14336 N4096 19.1 -> 17.4, M512 K2048 N4096 14.4 -> 13.0 (each as it was then).
  programmatic_begin();
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const int x_rows = p.row_tile / CG;                  // activation rows this CTA stages
  const uint32_t x_half = uint32_t(x_rows) * 128u;     // one box of 64 k
  const uint32_t smem_x = base;
  const uint32_t smem_w = smem_x + uint32_t(p.x_stages) * 2u * x_half;
  const uint32_t bars = smem_w + uint32_t(p.w_stages) * W_STAGE;
  const uint32_t full_w = bars;                        // [w_stages] packed words and scales landed
  const uint32_t empty_w = full_w + 8 * p.w_stages;    // [w_stages] read by the dequantisers
  // One pair of barriers per k block in flight (block i: number i % x_stages) covers both operands: its activations lie
  // in stage i % x_stages of shared memory, its expanded weights in stage i % A_STAGES of tensor memory.
  const uint32_t full = empty_w + 8 * p.w_stages;      // [x_stages] leader: activations landed, expanded weights stored
  const uint32_t empty = full + 8 * p.x_stages;        // [x_stages] MMAs done with them
  const uint32_t tmem_full = empty + 8 * p.x_stages;   // [2 and the last tile's; RING] accumulators complete
  const uint32_t tmem_empty = tmem_full + 8 * RING;    // [2; RING] leader: accumulators drained
  const uint32_t tmem_slot = tmem_empty + 8 * RING;
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(base_ptr + (tmem_slot - base));
  const uint32_t parts_full = tmem_slot + 8;           // split: the partial sums of this CTA's rows have arrived
  // grouped: {expert, rows in use} of this CTA's items, or of every tile where those are fewer
  int2* list = reinterpret_cast<int2*>(base_ptr + (tmem_slot - base) + 16);

  const int tid = threadIdx.x;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // known to be uniform
  const int lane = tid & 31;
  const int rank = CG == 2 || p.split > 1 ? int(cluster_rank()) : 0;
  const bool leader = CG == 1 || rank == 0;

  if (warp == 0) {          // a lane per stage (at most 16 of a kind)
    if (lane == 0) {
      prefetch_tensormap(&map_w);
      prefetch_tensormap(&map_s);
      prefetch_tensormap(&map_x);
      mbar_init(parts_full, 1);
    }
    if (lane < p.w_stages) {
      mbar_init(full_w + 8 * lane, 1);
      mbar_init(empty_w + 8 * lane, MODE == MODE_SKINNY ? 8 : 4);   // (the epilogue reads the scales of a stage)
    }
    if (lane < p.x_stages) {
      mbar_init(full + 8 * lane, 4 * CG + 1);
      mbar_init(empty + 8 * lane, 1);
    }
    if (lane < RING) {
      mbar_init(tmem_full + 8 * lane, 1);
      mbar_init(tmem_empty + 8 * lane, 4 * CG);
    }
    fence_mbar_init();
  }
  if (warp == 1) {
    if (CG == 2) tmem_alloc_pair(tmem_slot, 512);
    else tmem_alloc(tmem_slot, 512);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();   // barriers are initialised before anything arrives remotely
  else if (p.split > 1) cluster_arrive();
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  // everything above is done while the kernel before is still at work, everything below may read what that one wrote
  programmatic_wait();
  int m_tiles = p.m_tiles;
  if (!dense_mode(MODE)) m_tiles = min(m_tiles, (*p.total_rows + 127) / 128);
  const int items = m_tiles * p.n_tiles;
  // split: the CTAs of a cluster (a row of the grid) work on one item, each on its own share of the k blocks
  const int first_item = p.split > 1 ? int(blockIdx.y) : int(blockIdx.x) / CG;
  const int item_step = p.split > 1 ? items : int(gridDim.x) / CG;
  const int kb_first = p.split > 1 ? rank * p.kb_each + min(rank, p.kb_extra) : 0;
  const int kb_count = p.kb_each + (p.split > 1 && rank < p.kb_extra ? 1 : 0);
  // item / d without a division (items * d < 2^32)
  auto tile_quotient = [&](int item) { return p.tile_magic ? int(__umulhi(uint32_t(item), p.tile_magic)) : item; };
  struct Item {
    int row0, n_tile, expert, rows, n;   // n: rows of the MMA, a multiple of 16 * CG
  };
  const int my_items = items > first_item ? (items - 1 - first_item) / item_step + 1 : 0;
  auto item_of = [&](int item, int local) {   // the local-th one of this CTA
    Item t;
    if (dense_mode(MODE)) {
      t.n_tile = tile_quotient(item);   // the row tile varies fastest
      const int m_tile = item - t.n_tile * m_tiles;
      t.row0 = m_tile * p.row_tile;
      t.expert = 0;
      t.rows = min(p.row_tile, p.M - t.row0);
    } else {
      const int tile = tile_quotient(item);   // the column tile varies fastest
      t.n_tile = item - tile * p.n_tiles;
      t.row0 = tile * 128;
      const int2 e = list[p.list_by_item ? local : tile];
      t.expert = e.x;
      t.rows = e.y;
    }
    t.n = max(16 * CG, (t.rows + 16 * CG - 1) / (16 * CG) * (16 * CG));
    return t;
  };

  if (!dense_mode(MODE)) {
    // Rows in use of a 128-row block: its routes come first, padding follows.  Bound by the latency of the loads, hence one
    // round of them, which does not wait for the number of rows: as a loop over all blocks, a warp and block at a time, this
    // took 17 of the 650 us of the up|gate contraction of 16384 tokens on 64 experts and 2 to 4 us at 64 tokens.
    const int per_expert = p.block_rows / 128;
    for (int e = warp; e < p.list_items; e += THREADS / 32) {
      const int tile = p.list_by_item ? tile_quotient(first_item + e * item_step) : e;
      if (tile >= p.m_tiles) break;
      int rows = min(128, p.M - tile * 128), expert = __ldg(p.tile_expert + tile / per_expert);
      if (p.row_route != nullptr) {
        int last = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = i * 32 + lane;
          const int route = r < rows ? __ldg(p.row_route + tile * 128 + r) : -1;
          const unsigned used = __ballot_sync(0xffffffffu, route >= 0 && route < p.routes);
          if (used) last = i * 32 + 32 - __clz(used);
        }
        rows = last;
      }
      if (lane == 0) {
        if (unsigned(expert) >= unsigned(p.experts)) {
          // an id that names no expert (a stale or sentinel table entry): never used as an index.  The plane past
          // the last expert reads as zeros: zero scales, so zero weights
          if (tile < m_tiles) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_INDEX);
          expert = p.experts;
        }
        list[e] = make_int2(expert, rows);
      }
    }
    __syncthreads();
  }

  // split: the rows of a tile are dealt out in slices of whole fours, one for each CTA of the cluster; a CTA sends its sums of
  // every slice to the CTA that owns it.  Its room there: [rank][four of rows][column], 16 bytes each, so that the lanes of
  // a warp write and read 512 bytes in a row.
  const uint32_t parts = base + p.exchange;
  bool waited = false;    // for the other CTAs of the cluster to be there
  auto slice_fours = [&](int fours) { return (fours + p.split - 1) / p.split; };
  auto send_part = [&](int four, int column, int fours, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
    const int slice = slice_fours(fours), owner = four / slice;
    const uint32_t to = parts + uint32_t((rank * slice + four - owner * slice) * COLS + column) * 16u;
    if (owner == rank)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(to), "r"(v0), "r"(v1), "r"(v2), "r"(v3) : "memory");
    else
      store_async_v4(map_to_rank(to, owner), v0, v1, v2, v3, map_to_rank(parts_full, owner));
  };

  if (warp == 0) {
    // ------------------------------ packed weights and scales ------------------
    const int scale_rows = BK >> p.group_shift;
    const uint32_t bytes = W_BYTES + uint32_t(scale_rows) * COLS * 2;
    const int tile_columns = MODE == MODE_UPGATE_SILU ? 64 : COLS, tile_rank = CG == 2 ? rank : 0;
    uint32_t s = 0, phase = 1;
    bool ok = true, ready = true;   // ready: the stage was seen to be free
    for (int item = first_item, local = 0; item < items && ok; item += item_step, ++local) {
      const Item t = item_of(item, local);
      const int column = (t.n_tile * CG + tile_rank) * tile_columns;
      int row = kb_first * W_ROWS, scale_row = kb_first * scale_rows;
      for (int kb = 0; kb < kb_count; ++kb, row += W_ROWS, scale_row += scale_rows) {
        const uint32_t bar = full_w + 8 * s, dst = smem_w + s * W_STAGE;
        ok = __all_sync(0xffffffffu, ready) || mbar_wait_warp(empty_w + 8 * s, phase);
        if (!ok) break;
        if (++s == uint32_t(p.w_stages)) s = 0, phase ^= 1;
        ready = mbar_test(empty_w + 8 * s, phase);
        if (elect_one()) {
          mbar_expect_tx(bar, bytes);
          tma_load_3d(dst, &map_w, column, row, t.expert, bar);
          tma_load_3d(dst + W_BYTES, &map_s, column, scale_row, t.expert, bar);
          if (MODE == MODE_UPGATE_SILU) {   // 64 gate columns, then the 64 up columns that go with them
            tma_load_3d(dst + W_BYTES / 2, &map_w, column + p.out_cols, row, t.expert, bar);
            tma_load_3d(dst + W_BYTES + scale_rows * 128, &map_s, column + p.out_cols, scale_row, t.expert, bar);
          }
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
  } else if (warp == 2) {
    // ------------------------------ activations --------------------------------
    const uint32_t full_leader = CG == 2 ? map_to_rank(full, 0) : full;
    uint32_t s = 0, phase = 1;
    bool ok = true, ready = true;
    for (int item = first_item, local = 0; item < items && ok; item += item_step, ++local) {
      const Item t = item_of(item, local);
      const int rows = t.n / CG, row0 = t.row0 + (CG == 2 ? rank * rows : 0);
      const int boxes = dense_mode(MODE) ? 1 : __shfl_sync(0xffffffffu, rows / 16, 0);
      const uint32_t bytes = uint32_t(CG * boxes * p.box_rows) * 256u;
      int k = kb_first * BK;
      for (int kb = 0; kb < kb_count; ++kb, k += BK) {
        const uint32_t own = full + 8 * s, bar = full_leader + 8 * s;
        uint32_t dst = smem_x + s * 2u * x_half;
        ok = __all_sync(0xffffffffu, ready) || mbar_wait_warp(empty + 8 * s, phase);
        if (!ok) break;
        if (++s == uint32_t(p.x_stages)) s = 0, phase ^= 1;
        ready = mbar_test(empty + 8 * s, phase);
        if (elect_one()) {
          if (leader) mbar_expect_tx(own, bytes);
          for (int box = 0, row = row0; box < boxes; ++box, row += 16, dst += 16 * 128) {
            if (CG == 2) {
              tma_load_2d_pair(dst, &map_x, k, row, bar);
              tma_load_2d_pair(dst + x_half, &map_x, k + 64, row, bar);
            } else {
              tma_load_2d(dst, &map_x, k, row, bar);
              tma_load_2d(dst + x_half, &map_x, k + 64, row, bar);
            }
          }
        }
        __syncwarp();
      }
    }
    if (!ok && lane == 0) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ---------------------------------
    // The whole warp walks the loop and one elected lane issues: with the loop inside `lane == 0` the descriptors live
    // in per-thread registers and every MMA takes about 60 cycles to issue, whatever its size.
    if (leader) {
      constexpr uint32_t fmt = std::is_same<T, __half>::value ? 0u : 1u;
      const bool issue = elect_one();
      const uint64_t desc_x = umma_desc_k_major_sw128(smem_x);
      const uint32_t desc_high = uint32_t(desc_x >> 32);
      uint32_t s = 0, phase = 0, a = 0, local = 0, ring = 0, ring_phase = 0;
      bool ok = true, ready = false;   // ready: both operands of the k block were seen to be there
      for (int item = first_item; item < items && ok; item += item_step, ++local) {
        const Item t = item_of(item, int(local));
        const uint32_t idesc = umma_idesc(1, fmt, fmt, 0, 0, CG * COLS, uint32_t(t.n));
        const uint32_t acc = p.acc_sets == 2 ? local & 1 : 0, use = p.acc_sets == 2 ? local >> 1 : local;
        if (MODE != MODE_SKINNY) {
          ok = mbar_wait_warp(tmem_empty + 8 * acc, (use & 1) ^ 1);
          if (!ok) break;
          tcgen05_fence_after();
        }
        const uint32_t tmem_d = tmem_base + acc * (ACC_COLUMNS / 2);
        for (int kb = 0; kb < kb_count; ++kb) {
          const uint32_t tmem_a = tmem_base + A_COLUMN + a * 64, done = empty + 8 * s;
          const uint32_t desc_low = uint32_t(desc_x) + s * (x_half >> 3);   // two halves of x_half / 16 units
          ok = __all_sync(0xffffffffu, ready) || mbar_wait_warp(full + 8 * s, phase);
          if (!ok) break;
          if (MODE == MODE_SKINNY) {
            ok = mbar_wait_warp(tmem_empty + 8 * ring, ring_phase ^ 1);
            if (!ok) break;
          }
          if (++s == uint32_t(p.x_stages)) s = 0, phase ^= 1;
          a = (a + 1) % A_STAGES;
          ready = mbar_test(full + 8 * s, phase);   // of the next k block
          tcgen05_fence_after();
          if (MODE == MODE_SKINNY) {
            if (issue) {
              const int steps = 1 << (p.group_shift - 4);   // MMAs of 16 k in a group
#pragma unroll
              for (int kk = 0; kk < 8; ++kk) {
                const uint32_t low = desc_low + (kk >= 4 ? (x_half >> 4) : 0u) + 2 * (kk & 3);
                umma_f16_ts<CG>(tmem_base + ring * GROUP_ACC + (kk >> (p.group_shift - 4)) * SKINNY_ROWS, tmem_a + kk * 8,
                                (uint64_t(desc_high) << 32) | low, idesc, (kk & (steps - 1)) != 0);
              }
              umma_commit(done);
              umma_commit(tmem_full + 8 * ring);
            }
            if (++ring == RING) ring = 0, ring_phase ^= 1;
          } else if (issue) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk) {   // 16 k: 8 columns of A, 32 bytes of a row of B
              const uint32_t low = desc_low + (kk >= 4 ? (x_half >> 4) : 0u) + 2 * (kk & 3);   // an address: no carry
              umma_f16_ts<CG>(tmem_d, tmem_a + kk * 8, (uint64_t(desc_high) << 32) | low, idesc, (kb | kk) != 0);
            }
            if (CG == 2) umma_commit_pair(done);
            else umma_commit(done);
          }
          __syncwarp();
        }
        if (MODE != MODE_SKINNY && ok && issue) {
          const uint32_t complete = tmem_full + 8 * (int(local) == my_items - 1 ? LAST_TILE : acc);
          if (CG == 2) umma_commit_pair(complete);
          else umma_commit(complete);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
    }
  } else if (MODE == MODE_UPGATE_SILU && warp == 3) {
    // ------------------------------ zeros for the kernel that adds to this buffer ----
    // Beside 600 us of contraction (16384 tokens of 4096: 268 MB), where a fill of its own takes 38.
    const int64_t step = int64_t(gridDim.x) * 128;
    for (int64_t at = int64_t(blockIdx.x) * 128; at < p.clear_vectors; at += step) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (at + i * 32 + lane < p.clear_vectors) p.clear[at + i * 32 + lane] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.clear_pause > 0) __nanosleep(p.clear_pause);
    }
  } else if (warp >= FIRST_DEQUANT) {
    // ------------------------------ dequantisers --------------------------------
    const int set = (warp - FIRST_DEQUANT) >> 2, quadrant = warp & 3;
    const uint32_t magic = Elem<T>::kMagic2 ^ (p.twos_complement ? 0x00080008u : 0u);
    const uint32_t flip = p.twos_complement ? 0x08080808u : 0u;
    // where this thread's column lies in a stage.  up|gate: a quadrant of lanes is 16 gate columns and the 16 up
    // columns that go with them, so that the gate is applied inside a warp
    uint32_t w_offset, w_pitch, s_offset, s_pitch;
    const uint32_t scale_rows = uint32_t(BK) >> p.group_shift;
    if (MODE == MODE_UPGATE_SILU) {
      const uint32_t column = quadrant * 16 + (lane & 15), up = uint32_t(lane) >> 4;
      w_pitch = 256, w_offset = up * (W_BYTES / 2) + column * 4;
      s_pitch = 128, s_offset = W_BYTES + up * (scale_rows * 128) + column * 2;
    } else {
      const uint32_t column = quadrant * 32 + lane;
      w_pitch = COLS * 4, w_offset = column * 4;
      s_pitch = COLS * 2, s_offset = W_BYTES + column * 2;
    }
    uint32_t s_of[4];   // scale of k 32 g .. 32 g + 31
#pragma unroll
    for (int g = 0; g < 4; ++g) s_of[g] = s_offset + (uint32_t(g * 32) >> p.group_shift) * s_pitch;
    const uint32_t total = uint32_t(my_items) * uint32_t(kb_count);
    const uint32_t tmem_a = tmem_base + A_COLUMN + set * 64 + (uint32_t(quadrant * 32) << 16);
    const uint32_t full_leader = CG == 2 ? map_to_rank(full, 0) : full;
    // A set always writes the same stage of tensor memory: free when the block A_STAGES before has been multiplied.
    // x is the barrier of the set's block, x_before that of its last one, A_STAGES before.
    uint32_t s = set, phase = 0, x = set, phase_x = 0, x_before = 0, phase_before = 0;
    bool ok = true;
    for (uint32_t i = set; i < total; i += SETS) {
      ok = mbar_wait_warp(full_w + 8 * s, phase);
      if (!ok) break;
      const uint32_t stage = smem_w + s * W_STAGE;
      uint32_t words[W_ROWS], scale[4];
#pragma unroll
      for (int r = 0; r < W_ROWS; ++r) words[r] = lds32(stage + w_offset + r * w_pitch);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const uint32_t v = MODE == MODE_SKINNY ? 0u : lds16(stage + s_of[g]);
        scale[g] = v | (v << 16);
      }
      // the words are in registers before the stage is handed back: the arrival waits for the loads it depends on
      asm volatile("" ::"r"(words[0]), "r"(words[W_ROWS - 1]), "r"(scale[3]) : "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(empty_w + 8 * s);
      s += SETS;
      if (s >= uint32_t(p.w_stages)) s -= p.w_stages, phase ^= 1;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t o[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint32_t w = words[half * 8 + j], scale2 = scale[half * 2 + (j >> 2)];
          if (MODE == MODE_SKINNY) {
            // A 16-bit integer q is the number q times the smallest subnormal, so that one multiply-add gives q - 8 exactly,
            // times a power of two.  The pairs come out of two masked words, a byte of zeros - the sign of a nibble - between.
            // 11 instructions a word instead of 13: M12 K4096 N14336 15.7 -> 15.3 us, M8 K8192 N8192 17.3 -> 16.7.  Weights
            // with their scale keep the other way: the scale times that power of two leaves the type's range (a half from 128
            // on, a bfloat16 from 2^122).  In bfloat16, with the factor in the scale / with a vote on the scales between the two
            // ways / so: M512 K2048 N4096 9.7 / 10.3 / 9.9 us, M24 K4096 N4096 7.05 / 7.45 / 7.20, 64 tokens on 64 experts 155.6 /
            // 160.0 / 156.8.
            const uint32_t even = lop3_and_xor_u32(w, 0x0F0F0F0Fu, flip), odd = lop3_and_xor_u32(w >> 4, 0x0F0F0F0Fu, flip);
            o[4 * j + 0] = prmt(even, odd, 0xC480);  // (k0, k1)
            o[4 * j + 1] = prmt(even, odd, 0xD591);  // (k2, k3)
            o[4 * j + 2] = prmt(even, odd, 0xE6A2);  // (k4, k5)
            o[4 * j + 3] = prmt(even, odd, 0xF7B3);  // (k6, k7)
          } else {
            const uint32_t w4 = w >> 4;
            o[4 * j + 0] = lop3_and_xor_u32(prmt(w, w4, 0x0400), 0x000F000Fu, magic);  // (k0, k1)
            o[4 * j + 1] = lop3_and_xor_u32(prmt(w, w4, 0x0501), 0x000F000Fu, magic);  // (k2, k3)
            o[4 * j + 2] = lop3_and_xor_u32(prmt(w, w4, 0x0602), 0x000F000Fu, magic);  // (k4, k5)
            o[4 * j + 3] = lop3_and_xor_u32(prmt(w, w4, 0x0703), 0x000F000Fu, magic);  // (k6, k7)
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (MODE == MODE_SKINNY) o[4 * j + c] = Elem<T>::tiny2(o[4 * j + c]);
            else o[4 * j + c] = Elem<T>::mul2(Elem<T>::sub2(o[4 * j + c], Elem<T>::kBias2), scale2);
          }
        }
        if (half == 0) {
          // The first half is expanded while the block that still lies in this stage is being multiplied.
#pragma unroll
          for (int j = 0; j < 32; ++j) asm volatile("" : "+r"(o[j]));
          if (i >= A_STAGES) ok = mbar_wait_warp(empty + 8 * x_before, phase_before);
          if (!ok) break;
          tcgen05_fence_after();
        }
        tmem_store_32x32(tmem_a + half * 32, o);
      }
      if (!ok) break;
      tmem_store_wait();
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_remote(full_leader + 8 * x);
        else mbar_arrive(full_leader + 8 * x);
      }
      x_before = x, phase_before = phase_x;
      x += SETS;
      if (x >= uint32_t(p.x_stages)) x -= p.x_stages, phase_x ^= 1;
    }
    if (!ok && lane == 0) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
  } else if (MODE == MODE_SKINNY && warp >= FIRST_EPILOGUE) {
    // ------------------------------ scaling and sum over the groups ------------
    const int quadrant = warp & 3, column = quadrant * 32 + lane, groups = BK >> p.group_shift;
    const uint32_t s_offset = W_BYTES + uint32_t(column) * 2;
    uint32_t s = 0, phase = 0, ring = 0, ring_phase = 0;
    bool ok = true;
    for (int item = first_item; item < items && ok; item += item_step) {
      const Item t = item_of(item, 0);
      float sum[SKINNY_ROWS];
#pragma unroll
      for (int r = 0; r < SKINNY_ROWS; ++r) sum[r] = 0.f;
      for (int kb = 0; kb < kb_count; ++kb) {
        ok = mbar_wait_warp(tmem_full + 8 * ring, ring_phase) && mbar_wait_warp(full_w + 8 * s, phase);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t stage = smem_w + s * W_STAGE + s_offset;
        const uint32_t taddr = tmem_base + ring * GROUP_ACC + (uint32_t(quadrant * 32) << 16);
        for (int g = 0; g < groups; ++g) {
          uint32_t v[SKINNY_ROWS];
          tmem_load_32x16(taddr + g * SKINNY_ROWS, v);
          const float scale = Elem<T>::to_float(uint16_t(lds16(stage + g * (COLS * 2))));
          tmem_load_wait();
#pragma unroll
          for (int r = 0; r < SKINNY_ROWS; ++r) sum[r] = fmaf(__uint_as_float(v[r]), scale, sum[r]);
        }
        tcgen05_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(tmem_empty + 8 * ring);
          mbar_arrive(empty_w + 8 * s);
        }
        if (++ring == RING) ring = 0, ring_phase ^= 1;
        if (++s == uint32_t(p.w_stages)) s = 0, phase ^= 1;
      }
      // the weights' power of two, at the end: a scale times it may leave the range of f32
#pragma unroll
      for (int r = 0; r < SKINNY_ROWS; ++r) sum[r] *= Elem<T>::kTinyScale;
      const int col = t.n_tile * COLS + column;
      if (p.split > 1) {
        cluster_wait();
        waited = true;
        if (ok)
#pragma unroll
          for (int g = 0; g < SKINNY_ROWS / 4; ++g)
            send_part(g, column, t.n / 4, __float_as_uint(sum[4 * g]), __float_as_uint(sum[4 * g + 1]),
                      __float_as_uint(sum[4 * g + 2]), __float_as_uint(sum[4 * g + 3]));
      } else if (ok && col < p.out_cols) {
        uint16_t* y = reinterpret_cast<uint16_t*>(p.y) + col;
#pragma unroll
        for (int r = 0; r < SKINNY_ROWS; ++r)
          if (r < t.rows) y[size_t(r) * p.out_cols] = Elem<T>::from_float(sum[r]);
      }
    }
    if (!ok && lane == 0) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
  }
  if (MODE != MODE_SKINNY && warp >= FIRST_EPILOGUE && (p.split == 1 || warp < FIRST_DEQUANT) && my_items > 0) {
    // ------------------------------ epilogue -----------------------------------
    // The dequantisers, whose work is done by then, take four fifths of the last tile: nothing is left to overlap it with.
    // Bound by the stores: two bytes a lane and four warps took 4 of the 13 us of a call of M512 K2048 N4096 (a tile a
    // CTA); eight bytes a lane and twenty warps, 13.06 -> 10.77 us.  That tile has a barrier of its own:
    // of tmem_full the dequantisers have seen no phase, and a wait by parity on a barrier that is two phases behind returns at
    // once (with fewer than four k blocks a tile, eight with one accumulator set, nothing else has them wait for the tiles before).
    const int quadrant = warp & 3, last = my_items - 1;
    const int share = warp >= FIRST_DEQUANT ? 1 + ((warp - FIRST_DEQUANT) >> 2) : 0;
    uint16_t* y = reinterpret_cast<uint16_t*>(p.y);
    float* yf = reinterpret_cast<float*>(p.y);
    constexpr int CHUNK = MODE == MODE_UPGATE_SILU ? 16 : 32;   // rows at a time
    // Lane r of a chunk: where row r goes and with what weight, asked for a chunk ahead (two dependent loads took most of
    // the epilogue's time).
    int next_token = -1;
    float next_weight = 0.f;
    auto next_route = [&](const Item& t, int c) {
      next_token = -1;
      next_weight = 0.f;
      if (c + lane < t.rows) {
        const int route = __ldg(p.row_route + t.row0 + c + lane);
        if (route >= 0 && route < p.routes) {
          next_weight = __ldg(p.route_weight + route);
          next_token = route / p.top_k;
        }
      }
    };
    for (int local = share ? last : 0; local <= last; ++local) {
      const int item = first_item + local * item_step;
      const Item t = item_of(item, local);
      const uint32_t acc = p.acc_sets == 2 ? local & 1 : 0, use = uint32_t(p.acc_sets == 2 ? local >> 1 : local);
      const int step = local == last ? (1 + SETS) * CHUNK : CHUNK;
      if (MODE == MODE_DOWN_SCATTER) next_route(t, share * CHUNK);
      if (!mbar_wait_warp(tmem_full + 8 * (local == last ? LAST_TILE : acc), local == last ? 0 : use & 1)) {
        if (lane == 0) atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
        break;
      }
      if (p.split > 1) break;   // the partial sums of the cluster are put together below
      tcgen05_fence_after();
      const uint32_t taddr = tmem_base + acc * (ACC_COLUMNS / 2) + (uint32_t(quadrant * 32) << 16);
#pragma unroll 1
      for (int c = share * CHUNK; c < t.rows; c += step) {
        // Predicated, not branched: a branch a row keeps the work of different rows apart, and the epilogue of a tile with
        // few k blocks then takes longer than its MMAs (16384 tokens on 64 experts of 4096 x 1408: up|gate 807 -> 640 us).
        if (MODE == MODE_UPGATE_SILU) {
          // lanes 0..15 hold gate columns, lanes 16..31 the matching up columns: of 16 rows each takes eight
          const bool is_up = lane >= 16;
          const int col = (t.n_tile * CG + (CG == 2 ? rank : 0)) * 64 + quadrant * 16 + (lane & 15);
          uint32_t v[16];
          tmem_load_32x16(taddr + c, v);
          tmem_load_wait();
          float h[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, is_up ? v[i] : v[8 + i], 16);
            const float gv = __uint_as_float(is_up ? got : v[i]), uv = __uint_as_float(is_up ? v[8 + i] : got);
            h[i] = silu_times(gv, uv);  // one rounding
          }
#pragma unroll
          for (int i = 0; i < 8; i += 4) {
            const uint2 four = swap_rows(Elem<T>::pack2(h[i], h[i + 1]), Elem<T>::pack2(h[i + 2], h[i + 3]), lane);
            const int r = c + i + (lane & 3) + (is_up ? 8 : 0);
            if (r < t.rows) *reinterpret_cast<uint2*>(y + size_t(t.row0 + r) * p.out_cols + (col & ~3)) = four;
          }
        } else {
          const int col = (t.n_tile * CG + (CG == 2 ? rank : 0)) * COLS + quadrant * 32 + lane;
          uint32_t v[32];
          tmem_load_32x32(taddr + c, v);
          if (MODE == MODE_DOWN_SCATTER) {
            const int token = next_token;
            const float weight = next_weight;
            next_route(t, c + step);
            tmem_load_wait();
            // Four lanes swap four rows of their four columns, so that each adds 16 bytes of one row: adds of four bytes a
            // lane stop at 1 TB/s (16384 tokens on 64 experts, whole layer: 1493 us with them, 1400 so).
            const bool odd = lane & 1, upper = lane & 2;
            const int first_col = col & ~3, off = first_col < p.out_cols ? 0 : int(0x80000000);
            float* to = yf + first_col;
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
              const uint32_t got0 = __shfl_xor_sync(0xffffffffu, odd ? v[i] : v[i + 1], 1);
              const uint32_t got1 = __shfl_xor_sync(0xffffffffu, odd ? v[i + 2] : v[i + 3], 1);
              const uint32_t a0 = odd ? got0 : v[i], a1 = odd ? v[i + 1] : got0;          // row 0 or 1
              const uint32_t b0 = odd ? got1 : v[i + 2], b1 = odd ? v[i + 3] : got1;      // row 2 or 3
              const uint32_t got2 = __shfl_xor_sync(0xffffffffu, upper ? a0 : b0, 2);
              const uint32_t got3 = __shfl_xor_sync(0xffffffffu, upper ? a1 : b1, 2);
              const int row_token = __shfl_sync(0xffffffffu, token, i + (lane & 3)) | off;
              const float w = __shfl_sync(0xffffffffu, weight, i + (lane & 3));
              const float c0 = __fmul_rn(w, __uint_as_float(upper ? got2 : a0));
              const float c1 = __fmul_rn(w, __uint_as_float(upper ? got3 : a1));
              const float c2 = __fmul_rn(w, __uint_as_float(upper ? b0 : got2));
              const float c3 = __fmul_rn(w, __uint_as_float(upper ? b1 : got3));
              asm volatile(
                  "{\n\t.reg .pred p;\n\tsetp.ge.s32 p, %5, 0;\n\t"
                  "@p red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n\t}"
                  ::"l"(to + int64_t(row_token) * p.out_cols), "f"(c0), "f"(c1), "f"(c2), "f"(c3), "r"(row_token)
                  : "memory");
            }
          } else {
            tmem_load_wait();
            const int left = col < p.out_cols ? t.rows - c : 0;
            if (MODE == MODE_GROUPED_F32) {
              size_t at = size_t(t.row0 + c) * p.out_cols + col;
#pragma unroll
              for (int i = 0; i < 32; ++i, at += p.out_cols)
                if (i < left) yf[at] = __uint_as_float(v[i]);
            } else {
              uint16_t* to = y + size_t(t.row0 + c + (lane & 3)) * p.out_cols + (col & ~3);
#pragma unroll
              for (int i = 0; i < 32; i += 4, to += 4 * size_t(p.out_cols)) {
                const uint2 four = swap_rows(Elem<T>::pack2(__uint_as_float(v[i]), __uint_as_float(v[i + 1])),
                                             Elem<T>::pack2(__uint_as_float(v[i + 2]), __uint_as_float(v[i + 3])), lane);
                if (i + (lane & 3) < left) *reinterpret_cast<uint2*>(to) = four;
              }
            }
          }
        }
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0 && local < last) {
        if (CG == 2) mbar_arrive_remote(map_to_rank(tmem_empty + 8 * acc, 0));
        else mbar_arrive(tmem_empty + 8 * acc);
      }
    }
  }

  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (dense_mode(MODE) && CG == 1 && p.split > 1) {
    // Every CTA of the cluster holds a partial sum of the whole tile; its owner adds up a slice in rank order.  Bound by the
    // round trips between the SMs: plain remote stores, 96 bytes from lane to lane, between two cluster barriers took 5 of
    // the 17.3 us of a call of M77 K14336 N4096, 15.1 with these (M16 K4096 N4096 8.4 -> 7.8, M128 13.7 -> 11.1; the own slice
    // through the same asynchronous stores: 15.5, 7.7, 11.9, and M256 K8192 N4096 20.3 instead of 18.8).
    tcgen05_fence_after();
    if (!waited) cluster_wait();
    if (MODE != MODE_SKINNY && p.exchange == 0) cluster_sync();   // the MMAs of all CTAs are done with the operand stages
    const Item t = item_of(first_item, 0);
    const int fours = t.n / 4, slice = slice_fours(fours), mine = max(0, min(slice, fours - rank * slice));
    if (tid == 0) mbar_expect_tx(parts_full, uint32_t((p.split - 1) * mine * COLS) * 16u);
    if (MODE != MODE_SKINNY) {
      const uint32_t taddr = tmem_base + (uint32_t((warp & 3) * 32) << 16);
      for (int c = (warp >> 2) * 16; c < t.n; c += (THREADS / 128) * 16) {
        uint32_t v[16];
        tmem_load_32x16(taddr + c, v);
        tmem_load_wait();
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          send_part((c + i) / 4, (warp & 3) * 32 + lane, fours, v[i], v[i + 1], v[i + 2], v[i + 3]);
      }
    }
    cluster_arrive();
    if (MODE != MODE_SKINNY) __syncthreads();
    if (mbar_wait_warp_cluster(parts_full, 0)) {
      const float4* from = reinterpret_cast<const float4*>(base_ptr + p.exchange);
      uint16_t* y = reinterpret_cast<uint16_t*>(p.y);
      for (int i = tid; i < mine * COLS; i += THREADS) {   // a four of rows has four warps
        const int c = i % COLS, first = (rank * slice + i / COLS) * 4, row = first + (lane & 3);
        const int col = t.n_tile * COLS + (c & ~3);
        float4 sum = from[i];
        for (int other = 1; other < p.split; ++other) {
          const float4 v = from[other * slice * COLS + i];
          sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        const uint2 four = swap_rows(Elem<T>::pack2(sum.x, sum.y), Elem<T>::pack2(sum.z, sum.w), lane);
        if (row < t.rows && col < p.out_cols)
          *reinterpret_cast<uint2*>(y + size_t(t.row0 + row) * p.out_cols + col) = four;
      }
    } else if (lane == 0) {
      atomicExch(&g_w4a16_tmem_status, INTENT_B200_ERR_TIMEOUT);
    }
    tcgen05_fence_before();
    __syncthreads();
  }
  if (CG == 2) cluster_sync();   // the peer's shared memory and TMEM stay alive until both CTAs are done
  if (warp == 1) {
    tcgen05_fence_after();
    if (CG == 2) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
  if (CG == 1 && p.split > 1) cluster_wait();   // nothing of the other CTAs is on its way to this one's shared memory
}

int device_sms() {
  static int sms = [] {
    int device = 0, value = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&value, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    return value;
  }();
  return sms;
}

template <typename T, int MODE, int CG>
int launch(const TmemCall& q, cudaStream_t stream) {
  const int sms = device_sms();
  if (sms <= 0) return INTENT_B200_ERR_UNSUPPORTED;
  TmemParams p{};
  p.y = q.out;
  p.M = int(q.rows);
  p.K = int(q.K);
  p.WN = int(q.WN);
  p.out_cols = int(q.out_cols);
  p.k_blocks = int((q.K + BK - 1) / BK);
  p.row_tile = q.row_tile;
  p.m_tiles = int((q.rows + p.row_tile - 1) / p.row_tile);
  p.n_tiles = MODE == MODE_UPGATE_SILU ? int(q.out_cols / (64 * CG)) : int((q.out_cols + COLS * CG - 1) / (COLS * CG));
  p.box_rows = dense_mode(MODE) ? p.row_tile / CG : 16;
  p.acc_sets = p.row_tile <= 128 ? 2 : 1;
  p.split = q.split;
  p.group_shift = q.group_size == 32 ? 5 : q.group_size == 64 ? 6 : 7;
  p.twos_complement = q.zero_point == -1 ? 1 : 0;
  p.total_rows = q.total_rows;
  p.tile_expert = q.tile_expert;
  p.block_rows = q.block_rows;
  p.experts = int(q.experts);
  p.row_route = q.row_route;
  p.route_weight = q.route_weight;
  p.routes = int(q.routes);
  p.top_k = q.top_k;
  p.clear = reinterpret_cast<float4*>(q.clear);
  p.clear_vectors = q.clear ? q.clear_vectors : 0;
  if (p.row_tile % (16 * CG) != 0 || p.row_tile < 16 * CG || p.row_tile > 128 * CG) return INTENT_B200_ERR_UNSUPPORTED;
  if (p.split < 1 || p.split > 8 || (p.split > 1 && (!dense_mode(MODE) || CG != 1 || p.k_blocks < p.split)))
    return INTENT_B200_ERR_UNSUPPORTED;
  if (MODE == MODE_SKINNY && (p.row_tile != SKINNY_ROWS || p.M > SKINNY_ROWS)) return INTENT_B200_ERR_UNSUPPORTED;
  if (!dense_mode(MODE) && (p.m_tiles > LIST_BLOCKS || q.block_rows % 128 != 0 || p.row_tile != 128))
    return INTENT_B200_ERR_UNSUPPORTED;

  // Up to eight stages of activations: a stage comes back after its MMAs and a load from the L2, some 2000 cycles, of
  // which four k blocks cover no more than that.  The rest is a ring for the packed words, which come from HBM.
  const int64_t items = int64_t(p.m_tiles) * p.n_tiles, at_once = sms / CG;
  const int64_t most_items = (items + at_once - 1) / at_once;   // of a CTA or a pair
  p.list_by_item = most_items < p.m_tiles;
  p.list_items = dense_mode(MODE) ? 0 : int(p.list_by_item ? most_items : p.m_tiles);
  const int list_bytes = p.list_items * 8;
  const int x_stage = p.row_tile / CG * 256;
  // split: the partial sums of a cluster have room of their own where that leaves five stages of activations, and lie where
  // the operands were otherwise
  const int sums = p.split > 1 ? p.split * ((p.row_tile / 4 + p.split - 1) / p.split) * COLS * 16 : 0;
  int fixed = 1024 + 512 + list_bytes + sums;
  if (sums > 0 && fixed + 5 * x_stage + 9 * W_STAGE > SMEM_LIMIT) fixed -= sums;
  p.x_stages = 8;
  while (p.x_stages > A_STAGES && fixed + p.x_stages * x_stage + 9 * W_STAGE > SMEM_LIMIT) --p.x_stages;
  p.w_stages = (SMEM_LIMIT - fixed - p.x_stages * x_stage) / W_STAGE;
  if (p.w_stages > 16) p.w_stages = 16;
  // A set waits for the words of every SETS-th k block: that the stage's earlier words have landed follows for it from
  // the block 2 * SETS before having been multiplied, with fewer stages it would not (a wait by parity, two phases behind)
  if (p.w_stages < 2 * SETS) return INTENT_B200_ERR_UNSUPPORTED;
  const int smem = fixed + p.x_stages * x_stage + p.w_stages * W_STAGE, operands = p.x_stages * x_stage + p.w_stages * W_STAGE;
  if (sums > operands) return INTENT_B200_ERR_UNSUPPORTED;
  if (sums > 0 && fixed >= 1024 + 512 + sums) p.exchange = uint32_t(operands + 512);

  const CUtensorMapDataType type =
      std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const uint32_t box_cols = MODE == MODE_UPGATE_SILU ? 64 : COLS;
  const uint64_t E = uint64_t(q.experts), K = uint64_t(q.K), WN = uint64_t(q.WN);
  CUtensorMap map_x, map_w, map_s;
  if (!make_tensor_map_2d(&map_x, type, q.x, uint64_t(q.rows), K, K * 2, uint32_t(p.box_rows), 64,
                          CU_TENSOR_MAP_SWIZZLE_128B) ||
      !make_tensor_map_3d(&map_w, CU_TENSOR_MAP_DATA_TYPE_INT32, q.w, E, K / 8, WN, WN * 4, K / 8 * WN * 4, W_ROWS,
                          box_cols, CU_TENSOR_MAP_SWIZZLE_NONE) ||
      !make_tensor_map_3d(&map_s, type, q.s, E, K / uint64_t(q.group_size), WN, WN * 2,
                          K / uint64_t(q.group_size) * WN * 2, uint32_t(BK / q.group_size), box_cols,
                          CU_TENSOR_MAP_SWIZZLE_NONE))
    return INTENT_B200_ERR_UNSUPPORTED;

  // The limit belongs to the kernel, not to the launch: the same value from every call, so that no thread lowers it
  // between another one's request and its launch.
  auto kernel = w4a16_tmem_kernel<T, MODE, CG>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT);
  if (e != cudaSuccess) return cuda_status(e);
  const int64_t fastest = dense_mode(MODE) ? p.m_tiles : p.n_tiles;
  if (items * fastest >= (int64_t(1) << 32) || (p.split > 1 && items > 65535)) return INTENT_B200_ERR_UNSUPPORTED;
  p.tile_magic = fastest == 1 ? 0u : uint32_t(((uint64_t(1) << 32) + fastest - 1) / fastest);
  p.kb_each = p.k_blocks / p.split;
  p.kb_extra = p.k_blocks % p.split;
  const int cluster = p.split > 1 ? p.split : CG;
  const int grid = int(p.split > 1 ? items * p.split : CG * (items < at_once ? items : at_once));
  if (LaunchFacts* sink = observe_sink())
    return record_launch(sink, reinterpret_cast<const void*>(kernel),
                         MODE == MODE_SKINNY ? (p.split > 1 ? "w4a16_tmem_kernel 16 rows, scaled in f32, k split over a cluster"
                                                            : "w4a16_tmem_kernel 16 rows, scaled in f32")
                         : CG == 2       ? "w4a16_tmem_kernel CTA pairs, 256 columns"
                         : p.split > 1 ? "w4a16_tmem_kernel k split over a cluster, 128 columns"
                                       : "w4a16_tmem_kernel single CTA, 128 columns",
                         grid, THREADS, smem, cluster);
  if (p.clear_vectors > 0) {
    // The warp that clears writes a piece of 2 KiB in 60 ns, and pauses so that it is done in about half of the contraction, a
    // k block of which takes 300 (`least`: tiles that the routes fill at least).  Where that is too short for it, because the
    // experts are narrow or the tiles few, a fill ahead of the launch is faster.  Whole layer, us, pause 0 / 50 / 200 / fill ahead:
    // 16384 tokens of 4096 on 64 experts of 128 columns 509 / 506 / 633 / 506, of 256 (one choice) 327 / 318 / 451 / 325, of
    // 512 665 / 688 / 707 / 727; 16384 of 8192, 8 of 128 (one choice) 536 / 555 / 843 / 523; 1024 of 4096, 2 of 128 (one choice)
    // 42 / 59 / 127 / 40; 256 on 8 of 128 32.9 / 32.0 / 41.4 / 35.9.  From 1024 columns on the pause makes no difference.
    const int64_t at_a_time = int64_t(grid) * 128, pieces = (p.clear_vectors + at_a_time - 1) / at_a_time;
    const int64_t least = std::min(items, (q.routes + 127) / 128 * p.n_tiles);
    const double contraction = 300.0 * double(p.k_blocks) * double((least + at_once - 1) / at_once);
    const double fill = 60.0 * double(pieces), ahead = 1000.0 + double(p.clear_vectors) * 16.0 / 7000.0;
    if (fill > contraction + ahead) {
      const cudaError_t filled = cudaMemsetAsync(p.clear, 0, size_t(p.clear_vectors) * 16, stream);
      if (filled != cudaSuccess) return cuda_status(filled);
      p.clear_vectors = 0;
    } else {
      p.clear_pause = int(std::min(50.0, std::max(0.0, (0.6 * contraction - fill) / double(pieces))));
    }
  }
  const dim3 ctas = p.split > 1 ? dim3(unsigned(p.split), unsigned(items), 1) : dim3(unsigned(grid), 1, 1);
  e = launch_w4a16(kernel, ctas, THREADS, smem, stream, cluster, map_x, map_w, map_s, p);
  if (e != cudaSuccess) return cuda_status(e);
  note_launch();
  return launch_status();
}

}  // namespace

template <typename T>
int w4a16_tmem(const TmemCall& q, int mode, bool pairs, cudaStream_t stream) {
  switch (mode) {
    case MODE_DENSE: return pairs ? launch<T, MODE_DENSE, 2>(q, stream) : launch<T, MODE_DENSE, 1>(q, stream);
    case MODE_SKINNY: return launch<T, MODE_SKINNY, 1>(q, stream);
    case MODE_UPGATE_SILU:
      return pairs ? launch<T, MODE_UPGATE_SILU, 2>(q, stream) : launch<T, MODE_UPGATE_SILU, 1>(q, stream);
    case MODE_GROUPED_F32:
      return pairs ? launch<T, MODE_GROUPED_F32, 2>(q, stream) : launch<T, MODE_GROUPED_F32, 1>(q, stream);
    case MODE_DOWN_SCATTER:
      return pairs ? launch<T, MODE_DOWN_SCATTER, 2>(q, stream) : launch<T, MODE_DOWN_SCATTER, 1>(q, stream);
  }
  return INTENT_B200_ERR_UNSUPPORTED;
}
template int w4a16_tmem<__half>(const TmemCall&, int, bool, cudaStream_t);
template int w4a16_tmem<__nv_bfloat16>(const TmemCall&, int, bool, cudaStream_t);

// Reads and clears this file's status word (the device is idle when it is called).
int w4a16_tmem_take_status(int* value) {
  int zero = 0;
  cudaError_t e = cudaMemcpyFromSymbol(value, g_w4a16_tmem_status, sizeof(int));
  if (e != cudaSuccess) return cuda_status(e);
  if (*value != 0) cudaMemcpyToSymbol(g_w4a16_tmem_status, &zero, sizeof(int));
  return INTENT_B200_OK;
}

}  // namespace ib200
