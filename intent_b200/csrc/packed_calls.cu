// The program entries behind one signature: a call is an array of 64-bit slots in the entry's own order (pointers,
// extents, strides, constants, workspace, stream).  A host that dispatches many entries (csrc/host/binder.cpp) needs
// neither a prototype per entry nor a foreign-function library.
#include <cstring>
#include <utility>

#include "common.cuh"

namespace ib200 {
namespace {

template <typename A>
A from_slot(int64_t slot) {
  if constexpr (std::is_pointer<A>::value) return reinterpret_cast<A>(slot);
  else return static_cast<A>(slot);
}

template <auto F>
struct Packed;
template <typename... A, int (*F)(A...)>
struct Packed<F> {
  static constexpr int slots = int(sizeof...(A));
  template <std::size_t... I>
  static int spread(const int64_t* s, std::index_sequence<I...>) { return F(from_slot<A>(s[I])...); }
  static int call(const int64_t* s) { return spread(s, std::index_sequence_for<A...>{}); }
  static_assert(((std::is_pointer<A>::value || std::is_integral<A>::value) && ...), "slots are integers and pointers");
};

struct Row {
  const char* name;
  int (*call)(const int64_t*);
  int slots;
};
#define IB200_PACKED(NAME) {#NAME, &Packed<&NAME>::call, Packed<&NAME>::slots}
const Row kRows[] = {
    IB200_PACKED(intent_b200_bf16_gemm),
    IB200_PACKED(intent_b200_bitnet_int2_matmul),
    IB200_PACKED(intent_b200_dequant_bf16_fp4_matmul),
    IB200_PACKED(intent_b200_gemm_f16),
    IB200_PACKED(intent_b200_gemm_i8),
    IB200_PACKED(intent_b200_moe_align_routes),
    IB200_PACKED(intent_b200_moe_combine),
    IB200_PACKED(intent_b200_moe_count_routes),
    IB200_PACKED(intent_b200_moe_expert_ffn_bf16),
    IB200_PACKED(intent_b200_moe_expert_ffn_f16),
    IB200_PACKED(intent_b200_moe_gather_routed_rows),
    IB200_PACKED(intent_b200_moe_gather_rows),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_f32_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_f32_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_f32_tiled_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_f32_tiled_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_scatter_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_scatter_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_scatter_tiled_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_down_scatter_tiled_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_clear_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_clear_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_routed_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_routed_f16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_tiled_bf16),
    IB200_PACKED(intent_b200_moe_grouped_w4a16_upgate_silu_tiled_f16),
    IB200_PACKED(intent_b200_moe_mark_expert_blocks),
    IB200_PACKED(intent_b200_moe_prefix_routes),
    IB200_PACKED(intent_b200_moe_route_positions),
    IB200_PACKED(intent_b200_moe_route_top2),
    IB200_PACKED(intent_b200_moe_scatter_routes),
    IB200_PACKED(intent_b200_quantized_gemm_f16),
    IB200_PACKED(intent_b200_quantized_projection),
    IB200_PACKED(intent_b200_ragged_grouped_gemm_bf16),
    IB200_PACKED(intent_b200_ragged_grouped_gemm_f16),
    IB200_PACKED(intent_b200_routed_expert_projection_bf16),
    IB200_PACKED(intent_b200_routed_expert_projection_f16),
    IB200_PACKED(intent_b200_w4a16_gemm_bf16),
    IB200_PACKED(intent_b200_w4a16_gemm_f16),
    IB200_PACKED(intent_b200_w4a16_gemm_tiled_bf16),
    IB200_PACKED(intent_b200_w4a16_gemm_tiled_f16),
    IB200_PACKED(intent_b200_w4a16_gemv_bf16),
    IB200_PACKED(intent_b200_w4a16_gemv_f16),
    IB200_PACKED(intent_b200_w4a8_packed_matmul),
    IB200_PACKED(intent_b200_w8a8_gemm_bf16),
    IB200_PACKED(intent_b200_weight_only_int4_matmul_bf16),
    IB200_PACKED(intent_b200_weight_only_int4_matmul_f16),
};

}  // namespace
}  // namespace ib200

// The packed form of the program entry `name` and its number of slots; null when there is none.
extern "C" intent_b200_packed_fn intent_b200_packed_call(const char* name, int32_t* slots) {
  for (const auto& row : ib200::kRows)
    if (name && std::strcmp(row.name, name) == 0) {
      if (slots) *slots = row.slots;
      return row.call;
    }
  return nullptr;
}
