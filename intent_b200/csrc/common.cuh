// Shared host/device helpers of the sm_100a quantized-contraction library.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "../../include/intent_b200.h"

namespace ib200 {

// ---- host side -----------------------------------------------------------

// Process-wide count of kernels launched by this library.
void note_launch(int count = 1);

// The status of a CUDA call.  An error that is returned is not left for the next caller who asks for the last one.
inline int cuda_status(cudaError_t error) {
  if (error == cudaSuccess) return INTENT_B200_OK;
  cudaGetLastError();
  return INTENT_B200_ERR_CUDA + static_cast<int>(error);
}

// Returns the status of the launch that was just issued (cudaPeekAtLastError
// would also see sticky errors of unrelated work; cudaGetLastError clears ours).
inline int launch_status() { return cuda_status(cudaGetLastError()); }

// Dry-run observation of a launch: while a sink is installed on the calling thread (intent_b200_observe_begin),
// the main compute kernels' launch sites fill it with what they WOULD launch - the kernel instance's resource
// usage from cudaFuncGetAttributes and the launch plan - and launch nothing.
struct LaunchFacts {
  int valid;
  int registers;        // per thread
  int local_bytes;      // per-thread local memory (register spills land here)
  int static_smem;      // bytes
  int dynamic_smem;     // bytes requested by this launch
  int threads;          // per CTA
  int grid;             // CTAs
  int cluster;          // CTAs per cluster (1 = none)
  char kernel[64];      // kernel family and the plan's distinguishing choice
};
LaunchFacts* observe_sink();

// The process-wide switches that change which kernel or which plan an entry selects, in one place: what a launch was
// selected by can be kept as one copy, and a dry run on behalf of that launch selects by the copy.
struct Selection {
  int32_t gemm_pairs = 1;        // dense W4A16: CTA pairs may be chosen
  int32_t stream_grid = 0;       // bandwidth kernel: CTAs (0 = one per SM)
  int32_t stream_warps = 0;      // bandwidth kernel: warps (0 = built-in choice)
  int32_t table_ride = 1;        // 0 forces the staged form (measurement and tests)
  int32_t table_single = 1;      // a single small problem runs as a table of one (0 = never; for measurement)
  int32_t table_unit_rows = 0;   // 64 = the ride-along form uses 64-row units for problems of up to four rows; for measurement
  int32_t table_corr_mma = -1;   // ride-along kernel: correction sums by MMA (1), from the activations (0), built-in choice (-1)
  int32_t table_slots = 0;       // upper limit on the ring's slots (0 = the built-in choice); for measurement
};
Selection& process_selection();      // the switches themselves
const Selection& selection();        // what the call at hand selects by: the switches, or the copy of the launch observed
int record_launch(LaunchFacts* sink, const void* kernel, const char* name, int grid, int threads, int dynamic_smem,
                  int cluster);

struct View2 {
  void* p;
  int64_t d0, d1, s0, s1;
};
struct View1 {
  void* p;
  int64_t d0, s0;
};
struct View3 {
  void* p;
  int64_t d0, d1, d2, s0, s1, s2;
};

inline bool contiguous(const View1& v) { return v.d0 <= 1 || v.s0 == 1; }
inline bool contiguous(const View2& v) {
  return (v.d1 <= 1 || v.s1 == 1) && (v.d0 <= 1 || v.s0 == v.d1);
}
inline bool contiguous(const View3& v) {
  return (v.d2 <= 1 || v.s2 == 1) && (v.d1 <= 1 || v.s1 == v.d2) && (v.d0 <= 1 || v.s0 == v.d1 * v.d2);
}
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// A programmatic launch: the kernel may start on SMs that the kernel ahead of it has left, and waits inside
// (programmatic_wait) for everything ahead of it in the stream before it touches global memory.  What it does before that -
// barriers, tensor memory, indexes - and the launch itself then cost nothing beside the kernel ahead.
template <typename... P, typename... A>
cudaError_t launch_early(bool early, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                         const A&... arguments) {
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = block;
  config.dynamicSmemBytes = smem;
  config.stream = stream;
  cudaLaunchAttribute attribute[2];
  attribute[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
  attribute[1].id = cudaLaunchAttributeClusterDimension;
  attribute[1].val.clusterDim.x = unsigned(cluster);
  attribute[1].val.clusterDim.y = 1;
  attribute[1].val.clusterDim.z = 1;
  config.attrs = attribute;
  config.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<P>(arguments)...);
}

// Whether a bandwidth or table launch asks for its weights before its own wait (w4a16_stream.cu, w4a16_table.cu).
bool overlap_switched();

// For the W4A16 kernels of few rows and those with the weights in tensor memory, a row of which such a launch may overtake.
template <typename... P, typename... A>
cudaError_t launch_w4a16(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                         const A&... arguments) {
  return launch_early(true, kernel, grid, block, smem, stream, cluster, arguments...);
}

// For all others: with the switch on these start when all ahead of them has completed, so that the launch behind them cannot
// overtake what wrote its weights.  (To let it start only after their own wait costs small chains 1 us: an MoE layer's call 25.3
// -> 26.3 us.)
template <typename... P, typename... A>
cudaError_t launch_programmatic(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster,
                                const A&... arguments) {
  return launch_early(!overlap_switched(), kernel, grid, block, smem, stream, cluster, arguments...);
}

#define IB200_VIEW1_ARG(p) ib200::View1{p, p##_d0, p##_s0}
#define IB200_VIEW2_ARG(p) ib200::View2{p, p##_d0, p##_d1, p##_s0, p##_s1}
#define IB200_VIEW3_ARG(p) ib200::View3{p, p##_d0, p##_d1, p##_d2, p##_s0, p##_s1, p##_s2}

// ---- device side ---------------------------------------------------------
#ifdef __CUDACC__

// lets the next programmatic launch start as soon as every CTA of this one has
__device__ __forceinline__ void programmatic_begin() { asm volatile("griddepcontrol.launch_dependents;"); }
// everything ahead in the stream has completed and its writes are visible
__device__ __forceinline__ void programmatic_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ uint32_t lop3_and_or(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));  // (a & b) | c
  return d;
}

__device__ __forceinline__ uint32_t lop3_and_xor_u32(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(d) : "r"(a), "r"(b), "r"(c));  // (a & b) ^ c
  return d;
}

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t selector) {
  uint32_t d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
  return d;
}

__device__ __forceinline__ uint4 ldg_stream_v4(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ uint2 ldg_stream_v2(const void* p) {
  uint2 v;
  asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
  return v;
}

// silu(gate) * up in f32.  The hardware's reciprocal is off by up to one unit in the last place; one step of Newton's
// iteration rounds it as a division would, without the branch per value that a division has, which kept the values of a thread
// from overlapping (16384 tokens on 64 experts: up|gate 807 -> 640 us).  The bits of all 2^32 gates are those of
// gate * __frcp_rn(1 + __expf(-gate)); without the step 41 million of them differed, and the rms error against 64 bits was 3.3233e-7
// in place of 3.3157e-7.
__device__ __forceinline__ float silu_times(float gate, float up) {
  const float d = 1.0f + __expf(-gate);
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(r, fmaf(-fminf(d, 3.402823466e38f), r, 1.0f), r);   // (of infinity: zero)
  return gate * r * up;
}

// Element-type traits for the 16-bit activation types.
template <typename T>
struct Elem;

template <>
struct Elem<__half> {
  // 0x6400 | q is the half 1024 + q (ulp is 1 at 2^10); subtracting 1032 gives q - 8 exactly.
  static constexpr uint32_t kMagic2 = 0x64006400u;
  static constexpr uint32_t kBias2 = 0x64086408u;  // half2(1032, 1032)
  // The bits q alone are the half q * 2^-24: times 2^15, less 2^-6, they give (q - 8) * 2^-9 exactly.
  __device__ static __forceinline__ uint32_t tiny2(uint32_t q) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(q), "r"(0x78007800u), "r"(0xA400A400u));
    return d;
  }
  static constexpr float kTinyScale = 512.f;
  __device__ static __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  __device__ static __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  __device__ static __forceinline__ float to_float(uint16_t bits) {
    return __half2float(__ushort_as_half(bits));
  }
  __device__ static __forceinline__ uint16_t from_float(float v) {
    return __half_as_ushort(__float2half_rn(v));
  }
  __device__ static __forceinline__ uint32_t pack2(float low, float high) {
    uint32_t d;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(high), "f"(low));
    return d;
  }
  __device__ static __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                  uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

template <>
struct Elem<__nv_bfloat16> {
  // 0x4300 | q is the bfloat16 128 + q (ulp is 1 at 2^7); subtracting 136 gives q - 8 exactly.
  static constexpr uint32_t kMagic2 = 0x43004300u;
  static constexpr uint32_t kBias2 = 0x43084308u;  // bf16x2(136, 136)
  // The bits q alone are the bfloat16 q * 2^-133: times 2^127, less 2^-3, they give (q - 8) * 2^-6 exactly.
  __device__ static __forceinline__ uint32_t tiny2(uint32_t q) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(q), "r"(0x7F007F00u), "r"(0xBE00BE00u));
    return d;
  }
  static constexpr float kTinyScale = 64.f;
  __device__ static __forceinline__ uint32_t sub2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  __device__ static __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
  }
  __device__ static __forceinline__ float to_float(uint16_t bits) {
    return __uint_as_float(static_cast<uint32_t>(bits) << 16);
  }
  __device__ static __forceinline__ uint16_t from_float(float v) {
    return __bfloat16_as_ushort(__float2bfloat16_rn(v));
  }
  __device__ static __forceinline__ uint32_t pack2(float low, float high) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(high), "f"(low));
    return d;
  }
  __device__ static __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                  uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

#endif  // __CUDACC__

// w4a16_table.cu: one small contraction as a table of one problem (kTableDeclined: not that kind of call)
constexpr int kTableDeclined = -77001;
int w4a16_table_single_f16(View2, View2, View2, View2, int, int, void*, int64_t, cudaStream_t);
int w4a16_table_single_bf16(View2, View2, View2, View2, int, int, void*, int64_t, cudaStream_t);
int64_t w4a16_table_single_workspace_bytes(int64_t M, int64_t K, int64_t N);

}  // namespace ib200
