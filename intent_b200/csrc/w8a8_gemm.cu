// int8 x int8 -> int32 GEMM on tcgen05 (kind::i8, s32 accumulation in TMEM).
//
// Programs:
//   gemm_i8    C[m,n] = i32(sum_k A[m,k] * B[k,n]) + bias[n]      (reference kernel body
//              examples/kernels/contraction/gemm.py:29-39; exact integer result)
//   w8a8_gemm  Y[m,n] = bf16( f32(acc[m,n]) * sa[m] * sb[n] )      (the benchmark's per-token x
//              per-channel epilogue on the same exact accumulator)
//
// A [M,K] is K-major and B [K,N] is N-major in HBM, exactly as the reference declares them;
// both go to shared memory unchanged through 128B-swizzled TMA boxes (A: 128 rows x 128 k,
// B: two boxes of 128 k rows x 128 columns) and the B operand is described to the tensor core
// as MN-major, so no transposition pass exists anywhere.  One persistent CTA per SM walks
// 128 x 256 tiles, or a pair of CTAs on neighbouring SMs 256 x 256 tiles (cta_group::2): warp 0
// issues TMA (4 stages of 48 KiB; pair: 6 of 32 KiB per CTA), one thread of warp 1 issues four
// K32 MMAs per stage, warps 2..5 drain the two TMEM accumulators.  What bounds it is the rate at
// which operands get into and out of shared memory; the pair reads two thirds of the bytes per
// operation.  4096 x 8192 x 8192 scaled, calls back to back: 214.7 -> 200.5 us (2.56 -> 2.74 POP/s).
// Calls with few tiles share a tile's k blocks among the CTAs of a cluster (split_k.cuh).
// With B_K_MAJOR the second operand is given as [N,K] (K contiguous, e.g. decoded packed weights)
// and is loaded as one 256-row K-major box.
// Every wait is bounded (see tma.cuh); a wait that gives up records a timeout status.
#include <algorithm>

#include "cluster.cuh"
#include "common.cuh"
#include "dense.cuh"
#include "split_k.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace ib200 {

__device__ int g_w8a8_gemm_status = 0;

namespace {

constexpr int BM = 128, BN = 256, BK = 128;
constexpr int A_BYTES = BM * BK;       // 16 KiB
constexpr int B_BOX_BYTES = BK * 128;  // one 128-column box, 16 KiB
constexpr int THREADS = 6 * 32;

// CG = CTAs that share a tile: 1 = 128 x 256, 2 = a pair on neighbouring SMs computes 256 x 256, each CTA holding its
// own 128 rows of A and half of the tile's B columns (32 KiB per k block and CTA instead of 48).
template <int CG>
struct Ring {
  static constexpr int STAGES = CG == 1 ? 4 : 6;
  static constexpr int B_BYTES = 2 * B_BOX_BYTES / CG;
  static constexpr int SMEM_BYTES = 1024 + STAGES * (A_BYTES + B_BYTES) + 256;
};

static_assert(Ring<1>::STAGES * (A_BYTES + Ring<1>::B_BYTES) >= kPartRoom, "the sums of a cluster lie where the operands were");

constexpr int64_t BAND_BYTES = int64_t(64) << 20;   // of A, from which on rows are walked in bands

struct I8Params {
  void* out;
  const int32_t* bias;      // gemm_i8 (may be null)
  const float* a_scales;    // w8a8
  const float* b_scales;
  int M, N, K;
  int k_blocks, m_tiles, n_tiles;
  int band;                 // row tiles of a band of the tile walk
  int split;                // CTAs of a cluster that share the k blocks of a tile (1 = none; lone tiles only)
};

// Tile walk: the row tile varies fastest, so that the columns of B in flight are few.  Where A is too large to stay in
// the L2 for a whole column of tiles, rows are walked in bands of 4096.  All rows / bands, us: 20720 x 6272 x 1840
// (130 MB of A) 240 / 189, 12384 x 7424 x 3664 (92 MB) 313 / 273, 24720 x 2816 x 1744 (70 MB) 181 / 173; but
// 9584 x 6656 x 2640 (64 MB) 151 / 160, and with two tiles per CTA the bands put full tiles behind full ones where the
// walk over all rows ends on the narrow last column: 7664 x 2048 x 544 25.2 / 29.9, 7072 x 800 x 1408 39.1 / 45.5.
__device__ __forceinline__ void tile_coords(int tile, const I8Params& p, int& m_tile, int& n_tile) {
  int first = 0, rows = p.m_tiles;
  if (p.band < p.m_tiles) {
    const int band = tile / (p.band * p.n_tiles);
    tile -= band * p.band * p.n_tiles;
    first = band * p.band;
    rows = min(p.band, p.m_tiles - first);
  }
  n_tile = tile / rows;
  m_tile = first + tile - n_tile * rows;
}

// EPILOGUE 0: bf16(acc * sa[m] * sb[n]);  1: int32 acc + bias[n]
// SPLIT: lone tiles, each shared by a cluster (an instance of its own: the other ones keep their registers)
template <int EPILOGUE, bool B_K_MAJOR, int CG, bool SPLIT = false>
__global__ void __launch_bounds__(THREADS, 1)
i8_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
               const I8Params p) {
  constexpr int STAGES = Ring<CG>::STAGES, B_BYTES = Ring<CG>::B_BYTES;
  extern __shared__ unsigned char smem_raw[];
  programmatic_begin();
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  unsigned char* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t smem_a = base;
  const uint32_t smem_b = smem_a + STAGES * A_BYTES;
  const uint32_t bars = smem_b + STAGES * B_BYTES;
  const uint32_t full = bars;
  const uint32_t empty = full + 8 * STAGES;
  const uint32_t tmem_full = empty + 8 * STAGES;
  const uint32_t tmem_empty = tmem_full + 16;
  const uint32_t tmem_slot = tmem_empty + 16;
  const uint32_t parts_full = tmem_slot + 8;   // split: the other CTAs' sums of this one's chunks have arrived
  volatile uint32_t* tmem_slot_ptr = reinterpret_cast<volatile uint32_t*>(base_ptr + (tmem_slot - base));

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int tiles = p.m_tiles * p.n_tiles;
  constexpr bool split = CG == 1 && SPLIT;
  const int rank = CG == 2 ? int(cluster_rank()) : 0;
  const SplitShare share{split ? int(cluster_rank()) : 0, p.split};
  // split: a row of the grid is a cluster, and has one tile
  const int first_tile = split ? int(blockIdx.y) : int(blockIdx.x) / CG, tile_step = split ? tiles : int(gridDim.x) / CG;
  const int kb_first = split ? share.first(p.k_blocks) : 0, kb_count = split ? share.count(p.k_blocks) : p.k_blocks;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full + 8 * s, 1);
      mbar_init(empty + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(tmem_full + 8 * s, 1);
      mbar_init(tmem_empty + 8 * s, 4 * CG);
    }
    mbar_init(parts_full, 1);
    fence_mbar_init();
  }
  if (warp == 1) {
    if (CG == 2) tmem_alloc_pair(tmem_slot, 512);
    else tmem_alloc(tmem_slot, 512);
  }
  tcgen05_fence_before();
  __syncthreads();
  if (CG == 2) cluster_sync();   // barriers of both CTAs are initialised before anything arrives remotely
  tcgen05_fence_after();
  const uint32_t tmem_base = *tmem_slot_ptr;
  programmatic_wait();

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int tile = first_tile; tile < tiles && ok; tile += tile_step) {
        int m_tile, n_tile;
        tile_coords(tile, p, m_tile, n_tile);
        for (int kb = kb_first; kb < kb_first + kb_count; ++kb, ++it) {
          const uint32_t s = it % STAGES;
          if (!mbar_wait(empty + 8 * s, ((it / STAGES) & 1) ^ 1)) { ok = false; break; }
          const int row0 = (m_tile * CG + rank) * BM, col0 = n_tile * BN + rank * (BN / CG);
          if (CG == 2) {   // the bytes of both CTAs complete on the leader's barrier
            if (rank == 0) mbar_expect_tx(full + 8 * s, 2 * (A_BYTES + B_BYTES));
            const uint32_t bar = map_to_rank(full + 8 * s, 0);
            tma_load_2d_pair(smem_a + s * A_BYTES, &map_a, kb * BK, row0, bar);
            if (B_K_MAJOR) tma_load_2d_pair(smem_b + s * B_BYTES, &map_b, kb * BK, col0, bar);
            else tma_load_2d_pair(smem_b + s * B_BYTES, &map_b, col0, kb * BK, bar);
            continue;
          }
          const uint32_t bar = full + 8 * s;
          mbar_expect_tx(bar, A_BYTES + B_BYTES);
          tma_load_2d(smem_a + s * A_BYTES, &map_a, kb * BK, row0, bar);
          if (B_K_MAJOR) {
            tma_load_2d(smem_b + s * B_BYTES, &map_b, kb * BK, col0, bar);
          } else {
            tma_load_2d(smem_b + s * B_BYTES, &map_b, col0, kb * BK, bar);
            tma_load_2d(smem_b + s * B_BYTES + B_BOX_BYTES, &map_b, col0 + 128, kb * BK, bar);
          }
        }
      }
      if (!ok) atomicExch(&g_w8a8_gemm_status, INTENT_B200_ERR_TIMEOUT);
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {   // the leader issues for the pair
      // s32 accumulator, signed 8-bit operands, A K-major, B MN-major (N contiguous)
      constexpr uint32_t idesc = umma_idesc(2, 1, 1, 0, B_K_MAJOR ? 0 : 1, CG * BM, BN);
      uint32_t it = 0, local = 0;
      bool ok = true;
      for (int tile = first_tile; tile < tiles && ok; tile += tile_step, ++local) {
        const uint32_t acc = local & 1;
        if (!mbar_wait(tmem_empty + 8 * acc, ((local >> 1) & 1) ^ 1)) { ok = false; break; }
        tcgen05_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BN;
        for (int kb = 0; kb < kb_count; ++kb, ++it) {
          const uint32_t s = it % STAGES;
          if (!mbar_wait(full + 8 * s, (it / STAGES) & 1)) { ok = false; break; }
          tcgen05_fence_after();
          const uint64_t desc_a = umma_desc_k_major_sw128(smem_a + s * A_BYTES);
          // 128-column spans are one box (16 KiB) apart, 8-row k groups 1 KiB apart
          const uint64_t desc_b = B_K_MAJOR ? umma_desc_k_major_sw128(smem_b + s * B_BYTES)
                                            : umma_desc_mn_major_sw128(smem_b + s * B_BYTES, B_BOX_BYTES);
#pragma unroll
          for (int kk = 0; kk < BK / 32; ++kk) {
            // A: 32 k = 32 bytes along its 128-byte row (2 units); B: 32 k rows of 128 bytes (256 units)
            const uint64_t a = desc_a + uint64_t(2 * kk), b = desc_b + uint64_t((B_K_MAJOR ? 2 : 256) * kk);
            if (CG == 2) umma_i8_pair(tmem_d, a, b, idesc, (kb | kk) != 0);
            else umma_i8(tmem_d, a, b, idesc, (kb | kk) != 0);
          }
          if (CG == 2) umma_commit_pair(empty + 8 * s);
          else umma_commit(empty + 8 * s);
        }
        if (ok) {
          if (CG == 2) umma_commit_pair(tmem_full + 8 * acc);
          else umma_commit(tmem_full + 8 * acc);
        }
      }
      if (!ok) atomicExch(&g_w8a8_gemm_status, INTENT_B200_ERR_TIMEOUT);
    }
  }
  // One chunk of 32 columns of a row
  auto finish = [&](const uint32_t (&v)[32], int row, float row_scale, int col) {
    if (row >= p.M) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int n0 = col + q * 8;
      if (n0 < p.N) {  // N is a multiple of 16
        if (EPILOGUE == 0) {
          const float4 s0 = __ldg(reinterpret_cast<const float4*>(p.b_scales + n0));
          const float4 s1 = __ldg(reinterpret_cast<const float4*>(p.b_scales + n0 + 4));
          const float sc[8] = {s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w};
          uint32_t o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float lo = (float(int32_t(v[8 * q + 2 * j])) * row_scale) * sc[2 * j];
            const float hi = (float(int32_t(v[8 * q + 2 * j + 1])) * row_scale) * sc[2 * j + 1];
            o[j] = uint32_t(__bfloat16_as_ushort(__float2bfloat16_rn(lo))) |
                   (uint32_t(__bfloat16_as_ushort(__float2bfloat16_rn(hi))) << 16);
          }
          *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + size_t(row) * p.N + n0) =
              make_uint4(o[0], o[1], o[2], o[3]);
        } else {
          int32_t* dst = reinterpret_cast<int32_t*>(p.out) + size_t(row) * p.N + n0;
          int4 b0 = make_int4(0, 0, 0, 0), b1 = make_int4(0, 0, 0, 0);
          if (p.bias) {
            b0 = __ldg(reinterpret_cast<const int4*>(p.bias + n0));
            b1 = __ldg(reinterpret_cast<const int4*>(p.bias + n0 + 4));
          }
          // integer addition wraps (two's complement), as the reference's numerics require
          *reinterpret_cast<uint4*>(dst) =
              make_uint4(v[8 * q + 0] + uint32_t(b0.x), v[8 * q + 1] + uint32_t(b0.y),
                         v[8 * q + 2] + uint32_t(b0.z), v[8 * q + 3] + uint32_t(b0.w));
          *reinterpret_cast<uint4*>(dst + 4) =
              make_uint4(v[8 * q + 4] + uint32_t(b1.x), v[8 * q + 5] + uint32_t(b1.y),
                         v[8 * q + 6] + uint32_t(b1.z), v[8 * q + 7] + uint32_t(b1.w));
        }
      }
    }
  };
  if (warp >= 2) {
    const int quadrant = warp & 3;
    uint32_t local = 0;
    for (int tile = first_tile; tile < tiles; tile += tile_step, ++local) {
      int m_tile, n_tile;
      tile_coords(tile, p, m_tile, n_tile);
      const uint32_t acc = local & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(tmem_full + 8 * acc, (local >> 1) & 1))) {
        if (lane == 0) atomicExch(&g_w8a8_gemm_status, INTENT_B200_ERR_TIMEOUT);
        break;
      }
      if (split) break;   // the partial sums of the cluster are put together below
      tcgen05_fence_after();
      const int row = (m_tile * CG + rank) * BM + quadrant * 32 + lane;
      const uint32_t taddr = tmem_base + acc * BN + (uint32_t(quadrant * 32) << 16);
      float row_scale = 0.f;
      if (EPILOGUE == 0 && row < p.M) row_scale = p.a_scales[row];
#pragma unroll 1
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t v[32];
        tmem_load_32x32(taddr + c * 32, v);
        tmem_load_wait();
        finish(v, row, row_scale, n_tile * BN + c * 32);
      }
      tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) {
        if (CG == 2) mbar_arrive_remote(map_to_rank(tmem_empty + 8 * acc, 0));
        else mbar_arrive(tmem_empty + 8 * acc);
      }
    }
  }

  __syncwarp();
  tcgen05_fence_before();
  __syncthreads();
  if (split) {
    tcgen05_fence_after();
    cluster_sync();   // the MMAs of all CTAs are done with the operand stages, where the sums go
    if (first_tile < tiles && warp >= 2) {
      int m_tile, n_tile;
      tile_coords(first_tile, p, m_tile, n_tile);
      const int quadrant = warp & 3, in_tile = quadrant * 32 + lane, row = m_tile * BM + in_tile;
      const int chunks = min(kPartChunks, (p.N - n_tile * BN + 31) / 32), warps = min(4, (p.M - m_tile * BM + 31) / 32);
      const uint32_t taddr = tmem_base + (uint32_t(quadrant * 32) << 16);
      const PartRoom room{smem_a, warps};
      if (warp == 2 && lane == 0) mbar_expect_tx(parts_full, expected_parts(share, chunks, warps));
      if (quadrant < warps) {
        send_parts(share, room, parts_full, taddr, chunks, quadrant, lane);
        if (mbar_wait_warp_cluster(parts_full, 0)) {
          float row_scale = 0.f;
          if (EPILOGUE == 0 && row < p.M) row_scale = p.a_scales[row];
          for (int c = share.rank; c < chunks; c += share.split) {
            uint32_t v[32];
            add_parts(share, room, taddr, c, quadrant, lane, [](uint32_t x, uint32_t y) { return x + y; }, v);
            finish(v, row, row_scale, n_tile * BN + c * 32);
          }
        } else if (lane == 0) {
          atomicExch(&g_w8a8_gemm_status, INTENT_B200_ERR_TIMEOUT);
        }
      }
    }
    __syncwarp();
    tcgen05_fence_before();
    cluster_sync();   // nothing is on its way to a CTA that is gone
  }
  if (CG == 2) cluster_sync();   // the peer's shared memory and TMEM stay alive until both CTAs are done
  if (warp == 1) {
    tcgen05_fence_after();
    if (CG == 2) tmem_dealloc_pair(tmem_base, 512);
    else tmem_dealloc(tmem_base, 512);
  }
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

struct I8Operands {
  View2 a, b;
  int64_t M, N, K;
};

template <int EPILOGUE, bool B_K_MAJOR, int CG>
int launch(const I8Operands& q, I8Params& p, int sms, cudaStream_t stream) {
  p.m_tiles = int((q.M + CG * BM - 1) / (CG * BM));
  p.n_tiles = int((q.N + BN - 1) / BN);
  p.band = q.M * q.K >= BAND_BYTES ? 32 / CG : p.m_tiles;   // 4096 rows
  CUtensorMap map_a, map_b;
  if (!make_tensor_map_2d(&map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, q.a.p, uint64_t(q.M), uint64_t(q.K), uint64_t(q.K), BM,
                          BK, CU_TENSOR_MAP_SWIZZLE_128B) ||
      !(B_K_MAJOR ? make_tensor_map_2d(&map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, q.b.p, uint64_t(q.N), uint64_t(q.K),
                                       uint64_t(q.K), BN / CG, BK, CU_TENSOR_MAP_SWIZZLE_128B)
                  : make_tensor_map_2d(&map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, q.b.p, uint64_t(q.K), uint64_t(q.N),
                                       uint64_t(q.N), BK, 128, CU_TENSOR_MAP_SWIZZLE_128B)))
    return INTENT_B200_ERR_UNSUPPORTED;
  const int tiles = p.m_tiles * p.n_tiles;
  p.split = CG == 1 && tiles <= 65535 ? split_of(tiles, p.k_blocks, q.M, B_K_MAJOR ? 0.25 : 0.45, sms) : 1;
  auto kernel = p.split > 1 ? i8_gemm_kernel<EPILOGUE, B_K_MAJOR, CG, CG == 1> : i8_gemm_kernel<EPILOGUE, B_K_MAJOR, CG, false>;
  constexpr int smem = Ring<CG>::SMEM_BYTES;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return cuda_status(e);
  const int grid = p.split > 1 ? tiles * p.split : CG * std::min(tiles, sms / CG);
  if (LaunchFacts* sink = observe_sink())
    return record_launch(sink, reinterpret_cast<const void*>(kernel),
                         CG == 2       ? "i8_gemm_kernel CTA pairs, 256x256 tiles"
                         : p.split > 1 ? "i8_gemm_kernel 128x256 tiles, k split over a cluster"
                                       : "i8_gemm_kernel 128x256 tiles, two accumulators",
                         grid, THREADS, smem, p.split > 1 ? p.split : CG);
  const dim3 ctas = p.split > 1 ? dim3(unsigned(p.split), unsigned(tiles), 1) : dim3(unsigned(grid), 1, 1);
  e = launch_programmatic(kernel, ctas, THREADS, smem, stream, p.split > 1 ? p.split : CG, map_a, map_b, p);
  if (e != cudaSuccess) return cuda_status(e);
  note_launch();
  return launch_status();
}

// Whether a call runs on CTA pairs.  A pair tile reads two thirds of the operand bytes per operation but covers 256
// rows: not where the 128-row tiles fill clearly fewer waves of the chip.  A pair launch also costs about 0.6 us more
// than a lone one, which a short walk does not earn back (graph replay, lone against pairs, us):
//   two tiles   M129 N256:    K1024 15.5 / 16.2, K4096 22.1 / 22.6, K8192 32.4 / 32.2
//   8 tiles     M129 N1024:   K1024 15.9 / 16.4, K3072 21.1 / 21.2, K4096 23.4 / 23.4, K8192 35.1 / 33.0
//   32 tiles    M512 N2048:   K1024 18.6 / 19.2, K1536 19.9 / 20.2, K2048 21.2 / 21.2, K4096 26.6 / 25.8
//   128 tiles   M1024 N4096:  K512 17.7 / 18.0, K1536 20.8 / 20.6, K4096 28.5 / 26.6
//   136 tiles   M2050 N2048:  K1536 19.4 / 19.7, K2048 21.0 / 21.1, K4096 26.6 / 25.8 (an odd row tile is half padding)
//   128 tiles   M2048 N2048:  K512 17.6 / 17.3, K1024 19.1 / 18.5, K4096 28.3 / 25.7 (many row tiles share B)
// so the k blocks that a pair walks, and those of the whole call, have to be enough.  How many is enough depends on
// the pitch of B's rows.  Boxes of 128 bytes on a pitch that is no multiple of 128 touch two lines of the L2 per row,
// and the half of B that a pair does not fetch weighs twice:
//   B [K,N]     M447 K4272 N1280 26.1 / 25.3, M319 K1728 N2816 19.6 / 20.6; M355 K4000 N2096 29.3 / 24.3
//   B [N,K]     M768 N3616: K3584 22.9 / 23.6; M1008 N4064: K7104 33.5 / 33.0; M816 N1168: K6496 30.2 / 26.4
// B [N,K] on lines of its own is fetched as one 256-row box by a lone CTA and gains nothing within one wave of pairs
// (M1616 K3328 N2064 19.3 / 20.1, M496 K8064 N2144 30.8 / 31.5); with several waves it does for long walks (two waves:
// M7104 K512 N624 15.4 / 15.8, M3248 K1280 N1392 19.9 / 19.3, M1776 K3840 N3040 35.2 / 32.2; more: M3568 K1536 N4784
// 42.8 / 45.7, M2992 K1792 N3840 38.3 / 36.9).  Nor do few columns, unless there are many row tiles to stream, which
// the deeper ring of a pair does better (N16: M4688 K5888 34.0 / 27.3, M7968 K5504 27.7 / 18.4, M2512 K6912 25.3 /
// 26.0).  And where the last wave of lone tiles is all in a narrow last column while that of the pairs is not, a short
// walk waits for the pairs' wide tiles (M1840 K1536 N7520 55.2 / 60.6, M825 K2080 N5472 29.8 / 35.6).
bool takes_pairs(int64_t M, int64_t N, int64_t K, bool b_k_major, int64_t sms) {
  if (M <= BM) return false;
  const int64_t k_blocks = (K + BK - 1) / BK;
  const int64_t row_tiles = (M + BM - 1) / BM, n_tiles = (N + BN - 1) / BN;
  const int64_t tiles = row_tiles * n_tiles, pair_tiles = (row_tiles + 1) / 2 * n_tiles;
  const int64_t waves = (tiles + sms - 1) / sms, pair_waves = (pair_tiles + sms / 2 - 1) / (sms / 2);
  if (pair_waves * 9 > waves * 10) return false;
  const int64_t walk = pair_waves * k_blocks, all = tiles * k_blocks;
  const int64_t tail = tiles - (waves - 1) * sms, pair_tail = pair_tiles - (pair_waves - 1) * (sms / 2);
  const bool narrow_end = N % BN > 0 && N % BN <= BN / 2 && tail <= row_tiles && pair_tail > (row_tiles + 1) / 2;
  if (pair_waves > 1 && narrow_end && k_blocks < 24) return false;
  const bool whole_lines = (b_k_major ? K : N) % 128 == 0;
  if (b_k_major) {
    if (pair_waves > 2) return k_blocks >= (whole_lines ? 16 : 10);
    if (N <= 32) return row_tiles >= 32;
    if (whole_lines) return pair_waves == 2 && k_blocks >= 10;
    if (N < 96 || (n_tiles == 1 && k_blocks < 32)) return false;   // little of B to share
  } else {
    if (pair_waves > 2 && k_blocks < 8) return false;
    if (whole_lines && pair_waves == 1) {
      if (n_tiles == 1) return false;
      if (K % 128 != 0) return k_blocks >= 32 && all >= 672;      // (the lines of A count on both forms)
      if (k_blocks >= 16)
        return (all >= 672 && (row_tiles > 2 || k_blocks >= 32)) || (k_blocks >= 48 && all >= 480);
    }
  }
  if (walk >= 16) return all >= 256;
  if (row_tiles % 2 != 0) return false;
  return pair_waves == 1 ? (k_blocks >= 12 && all >= 768) || (row_tiles >= 16 && tiles >= 112)
                         : pair_waves == 2 && row_tiles >= 16;
}

// b is [K,N] (N contiguous), or [N,K] (K contiguous) with B_K_MAJOR
template <int EPILOGUE, bool B_K_MAJOR = false>
int run(View2 a, View2 b, void* out, const int32_t* bias, const float* sa, const float* sb, cudaStream_t stream) {
  const int64_t M = a.d0, K = a.d1, N = B_K_MAJOR ? b.d0 : b.d1;
  if ((B_K_MAJOR ? b.d1 : b.d0) != K) return INTENT_B200_ERR_SHAPE;
  if (M == 0 || N == 0) return INTENT_B200_OK;
  if (!a.p || !b.p || !out) return INTENT_B200_ERR_NULL;
  if (!contiguous(a) || !contiguous(b)) return INTENT_B200_ERR_LAYOUT;
  if (!aligned16(a.p) || !aligned16(b.p) || !aligned16(out)) return INTENT_B200_ERR_LAYOUT;
  if (K == 0 || K % 16 != 0 || N % 16 != 0 || M > (1 << 24) || K > (1 << 24) || N > (1 << 24))
    return INTENT_B200_ERR_UNSUPPORTED;
  const int sms = device_sms();
  if (sms <= 0) return INTENT_B200_ERR_UNSUPPORTED;
  I8Params p{};
  p.out = out;
  p.bias = bias;
  p.a_scales = sa;
  p.b_scales = sb;
  p.M = int(M);
  p.N = int(N);
  p.K = int(K);
  p.k_blocks = int((K + BK - 1) / BK);
  const I8Operands q{a, b, M, N, K};
  if (sms >= 2 && takes_pairs(M, N, K, B_K_MAJOR, sms)) return launch<EPILOGUE, B_K_MAJOR, 2>(q, p, sms, stream);
  return launch<EPILOGUE, B_K_MAJOR, 1>(q, p, sms, stream);
}

}  // namespace

int i8_gemm_nt(const void* a, int64_t M, int64_t K, const void* b, int64_t N, int32_t* out, cudaStream_t stream) {
  View2 va{const_cast<void*>(a), M, K, K, 1}, vb{const_cast<void*>(b), N, K, K, 1};
  return run<1, true>(va, vb, out, nullptr, nullptr, nullptr, stream);
}

}  // namespace ib200

extern "C" int intent_b200_gemm_i8(INTENT_B200_VIEW2(a0), INTENT_B200_VIEW2(a1), INTENT_B200_VIEW1(a2),
                                   INTENT_B200_VIEW2(a3), void* stream) {
  using namespace ib200;
  if (a3_d0 != a0_d0 || a3_d1 != a1_d1 || a2_d0 != a1_d1) return INTENT_B200_ERR_SHAPE;
  if (!contiguous(IB200_VIEW2_ARG(a3)) || !contiguous(IB200_VIEW1_ARG(a2)) || !aligned16(a2)) return INTENT_B200_ERR_LAYOUT;
  return run<1>(IB200_VIEW2_ARG(a0), IB200_VIEW2_ARG(a1), a3, static_cast<const int32_t*>(a2), nullptr, nullptr,
                static_cast<cudaStream_t>(stream));
}

extern "C" int intent_b200_w8a8_gemm_bf16(INTENT_B200_VIEW2(a0), INTENT_B200_VIEW2(a1), INTENT_B200_VIEW1(a2),
                                          INTENT_B200_VIEW1(a3), INTENT_B200_VIEW2(a4), void* stream) {
  using namespace ib200;
  if (a4_d0 != a0_d0 || a4_d1 != a1_d1 || a2_d0 != a0_d0 || a3_d0 != a1_d1) return INTENT_B200_ERR_SHAPE;
  if (!contiguous(IB200_VIEW2_ARG(a4)) || !contiguous(IB200_VIEW1_ARG(a2)) || !contiguous(IB200_VIEW1_ARG(a3)) ||
      !aligned16(a2) || !aligned16(a3))
    return INTENT_B200_ERR_LAYOUT;
  if (a0_d0 > 0 && a1_d1 > 0 && (!a2 || !a3)) return INTENT_B200_ERR_NULL;
  return run<0>(IB200_VIEW2_ARG(a0), IB200_VIEW2_ARG(a1), a4, nullptr, static_cast<const float*>(a2),
                static_cast<const float*>(a3), static_cast<cudaStream_t>(stream));
}

extern "C" int intent_b200_i8_gemm_device_status(void) {
  int value = 0, zero = 0;
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return ib200::cuda_status(e);
  e = cudaMemcpyFromSymbol(&value, ib200::g_w8a8_gemm_status, sizeof(int));
  if (e != cudaSuccess) return ib200::cuda_status(e);
  if (value != 0) cudaMemcpyToSymbol(ib200::g_w8a8_gemm_status, &zero, sizeof(int));
  return value;
}
