// A 128 x 256 output tile whose k blocks are shared by the CTAs of a cluster (2, 4 or 8), each with a partial sum of the whole
// tile in its tensor memory.  The tile's chunks of 32 columns are dealt out in turn: a CTA sends its sums of every other
// chunk to the chunk's owner, 4 KiB a warp and chunk as one copy from shared memory to shared memory, and adds up its own in
// rank order.  (Asynchronous stores of 16 bytes a lane move a few bytes a nanosecond and SM: int8 M128 K4096 N4096 36 us with
// them, 14.0 so.)
//
// For calls with few tiles, which otherwise leave most SMs idle behind a long walk over k.  Whole tiles / split, us, calls one
// after another: int8 M26 K5520 N4336 31.7 / 14.6, M64 K8192 N1024 28.7 / 11.5, M100 K8192 N8192 37.3 / 22.9, M256 K2048
// N2048 17.1 / 12.9; B as [N,K] M20 K8192 N1024 24.7 / 12.5 (with the expansion before it); bf16 rows 95 and 32 of 2392 x 2104
// 26.2 / 15.6, 300 and 300 of 4096 x 1024 25.1 / 17.1; fp4 M3 K3840 N1328 25.4 / 14.5.
#pragma once

#include "cluster.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace ib200 {

constexpr int kPartChunks = 8;                  // of a tile
constexpr int kPartBytes = 32 * 32 * 4;         // a warp's 32 rows of a chunk
constexpr int kPartRoom = 192 * 1024;           // shared memory for the sums that are sent and those that arrive

// How many CTAs share a tile of up to `rows` rows: the least by estimate, in microseconds, `block` for 128 k of a lone tile
// (0.45; int8 rows of B in one box each 0.25) and 3 to 5 for the exchange, 1.5 more among eight.  What bounds the choice is
// room, for the clusters (clustered_ctas) and for the sums.
inline int split_of(int64_t tiles, int64_t k_blocks, int64_t rows, double block, int64_t sms) {
  const int64_t warps = rows >= 128 ? 4 : (rows + 31) / 32;
  int best = 1;
  double least = block * double(k_blocks);
  for (int split = 2; split <= 8; split *= 2) {
    if (tiles * split > clustered_ctas(split, sms) || k_blocks < 2 * split) break;
    if (2 * (kPartChunks - kPartChunks / split) * warps * kPartBytes > kPartRoom) break;
    const double cost = block * double((k_blocks + split - 1) / split) + 3.0 + 0.5 * double(warps) + (split == 8 ? 1.5 : 0.0);
    if (cost < least) least = cost, best = split;
  }
  return best;
}

#ifdef __CUDACC__

struct SplitShare {
  int rank, split;
  // k blocks of this CTA: the first `extra` ranks take one more
  __device__ __forceinline__ int first(int k_blocks) const { return rank * (k_blocks / split) + min(rank, k_blocks % split); }
  __device__ __forceinline__ int count(int k_blocks) const { return k_blocks / split + (rank < k_blocks % split ? 1 : 0); }
};

// Where the sums of a CTA's chunks arrive: [source, itself left out][chunk of the owner][quadrant of the rows], 4 KiB each;
// behind them those that it sends, [chunk][quadrant].  Inside: [four columns][row], 16 bytes each.
struct PartRoom {
  uint32_t base;
  int warps;      // quadrants of the tile that hold rows
  __device__ __forceinline__ uint32_t arriving(const SplitShare& share, int source, int owner, int chunk, int quadrant) const {
    const int per_owner = kPartChunks / share.split, place = source - (source > owner ? 1 : 0);
    return base + uint32_t(((place * per_owner + chunk / share.split) * warps + quadrant) * kPartBytes);
  }
  __device__ __forceinline__ uint32_t leaving(const SplitShare& share, int chunk, int quadrant) const {
    const int per_owner = kPartChunks / share.split;
    const int before = chunk - (chunk + share.split - 1 - share.rank) / share.split;   // chunks below that others own
    return base + uint32_t((((share.split - 1) * per_owner + before) * warps + quadrant) * kPartBytes);
  }
};

// One warp's 32 rows of the chunks that others own.  `chunks` of the tile lie in the matrix.
__device__ __forceinline__ void send_parts(const SplitShare& share, const PartRoom& room, uint32_t bar, uint32_t taddr, int chunks,
                                           int quadrant, int lane) {
#pragma unroll 1
  for (int c = 0; c < chunks; ++c) {
    const int owner = c % share.split;
    if (owner == share.rank) continue;
    uint32_t v[32];
    tmem_load_32x32(taddr + c * 32, v);
    tmem_load_wait();
    const uint32_t from = room.leaving(share, c, quadrant);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(from + uint32_t(i * 32 + lane) * 16u), "r"(v[4 * i]),
                   "r"(v[4 * i + 1]), "r"(v[4 * i + 2]), "r"(v[4 * i + 3])
                   : "memory");
    fence_proxy_async();
    __syncwarp();
    if (lane == 0)
      copy_to_cluster(map_to_rank(room.arriving(share, share.rank, owner, c, quadrant), owner), from, kPartBytes,
                      map_to_rank(bar, owner));
  }
}

// What arrives at a CTA when `warps` of the tile's four row quadrants hold rows.
__device__ __forceinline__ uint32_t expected_parts(const SplitShare& share, int chunks, int warps) {
  const int owned = (chunks - share.rank + share.split - 1) / share.split;
  return owned > 0 ? uint32_t((share.split - 1) * owned * warps * kPartBytes) : 0u;
}

// The sum over the cluster of an owned chunk, in rank order.
template <typename Add>
__device__ __forceinline__ void add_parts(const SplitShare& share, const PartRoom& room, uint32_t taddr, int chunk, int quadrant,
                                          int lane, Add add, uint32_t (&sum)[32]) {
  uint32_t own[32];
  tmem_load_32x32(taddr + chunk * 32, own);
  tmem_load_wait();
#pragma unroll 1
  for (int source = 0; source < share.split; ++source) {
    const uint32_t from = room.arriving(share, source, share.rank, chunk, quadrant);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint4 v = make_uint4(own[4 * i], own[4 * i + 1], own[4 * i + 2], own[4 * i + 3]);
      if (source != share.rank) v = lds128(from + uint32_t(i * 32 + lane) * 16u);
      sum[4 * i] = source == 0 ? v.x : add(sum[4 * i], v.x);
      sum[4 * i + 1] = source == 0 ? v.y : add(sum[4 * i + 1], v.y);
      sum[4 * i + 2] = source == 0 ? v.z : add(sum[4 * i + 2], v.z);
      sum[4 * i + 3] = source == 0 ? v.w : add(sum[4 * i + 3], v.w);
    }
  }
}

#endif  // __CUDACC__

}  // namespace ib200
