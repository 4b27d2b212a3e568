// Shared by the translation units of libflamia_b200.so.
#pragma once
#include "../../include/flamia_b200.h"
#include "sm100.cuh"

#include <utility>

namespace fl {

// cuTensorMapEncodeTiled, resolved at run time through the CUDA runtime (the library does not link libcuda, so it
// loads on a machine without a driver).
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn get_encode_tiled();

// 4-D map over a (b, s, heads, w) row-major byte tensor seen as dims {w, heads, s, b}; box {w, 1, rows, 1}.
// w bytes per row must be 32, 64 or 128 (one swizzle span).
int make_rows_map(CUtensorMap* m, const void* base, int b, int s, int heads, int w_bytes, int box_rows);
// same for 16-bit elements with w elements per row split into boxes of 64 elements (128 bytes): box {64, 1, rows, 1}
int make_rows_map_16(CUtensorMap* m, const void* base, int b, int s, int heads, int w_elems, int box_rows);
// (b, heads, s, w) layout (the f16 dQ accumulator): dims {w, s, heads, b}; box {64, rows, 1, 1}
int make_acc_map_16(CUtensorMap* m, const void* base, int b, int heads, int s, int w_elems, int box_rows);

int make_acc_t_map_16(CUtensorMap* m, const void* base, int b, int heads, int d, int s);

// FL_ERR_CUDA with the failing call and its CUDA code remembered for fl_last_cuda_error() (per host thread)
int cuda_fail(int cuda_code, const char* where);
// the result of a kernel launch just made: FL_OK, or cuda_fail() of cudaGetLastError()
int launch_result(const char* where);

// Allows a kernel `bytes` of dynamic shared memory on the current device. The attribute is set when a launch wants more than any
// before it and never lowered (setting it at every launch cost about a microsecond of host time each). FL_OK or cuda_fail().
int set_smem(const void* kern, int bytes, const char* where);
template <typename... A>
int set_smem(void (*kern)(A...), int bytes, const char* where) {
  return set_smem(reinterpret_cast<const void*>(kern), bytes, where);
}

// kern<<<grid, block, smem, st>>>(args...), started as soon as the blocks of the kernel ahead of it on the stream have left. Only for
// kernels that call grid_dependency() (sm100.cuh) before they touch global memory. (A step is six to nine launches with 1.5 to 2.5
// us between the end of one and the start of the next: b2 s2048 d96 window 512 step 117 -> 105 us, 6000 packed tokens 212 -> 196.)
template <typename... P, typename... A>
void launch_after(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);      // (launch_result() reports a failure)
}

// multiprocessors of the current device (cached per device): the size of a persistent grid
int sm_count();

// Division of n < 2^31 by a divisor known at launch: one multiplication (m = floor(2^(31 + l) / d) + 1 with 2^(l - 1) < d <= 2^l; the
// error n (m d - 2^(31 + l)) stays below 2^(31 + l)).
struct FastDiv {
  uint32_t m;
  int l, d;
  FastDiv() = default;
  explicit FastDiv(int div) : d(div) {
    for (l = 0; (1ll << l) < div; ++l) {}
    m = (uint32_t)((1ull << (31 + l)) / (uint32_t)div + 1);
  }
  __device__ __forceinline__ int div(int n) const { return (int)(((uint64_t)(uint32_t)n * m) >> (31 + l)); }
};

// A side of a sliding window (ABI: side + 1, 0 = unlimited) as the kernels take it: -1 = unlimited. A side beyond any sequence is cut,
// so that the kernels' sums of a position and a side stay inside 32 bits.
inline int window_side(int32_t p1) { return p1 <= 0 ? -1 : p1 - 1 < (1 << 30) ? p1 - 1 : (1 << 30); }

static constexpr long long kDefaultWaitCycles = 1ll << 31;

}  // namespace fl
