// Programmatic dependent launch.  A kernel launched with launch_pdl() may be scheduled while the
// kernel before it in the stream is still running; it must call pdl_wait() before it touches
// what that kernel may still be working on (the wait ends when every kernel before it has finished
// and its writes are visible).  A trigger lets the kernel after it start its own prologue.
// Launch latency and prologue (2-4 us of a kernel's ~10 on small frames) then overlap with the tail
// of the kernel before.
//
// A kernel that triggers does it behind its own wait, in one call (pdl_wait_and_trigger()), and a
// kernel launched this way leaves no CTA before its wait; the others' dependents start when they are
// over.  So when a kernel starts, all but the one launch directly before it are complete, and what those
// wrote may be read before pdl_wait(): the convolutions do.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace spconvb {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The kernel after this one may start once every CTA has been here.  (Nothing triggers without a wait:
// that kernel would start beside two others, and read what the first is still writing.)
__device__ __forceinline__ void pdl_wait_and_trigger() {
  asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;" ::: "memory");
}

// What an earlier kernel wrote, read where the source reads it: volatile, and through the coherent path.
// The compiler takes what __ldg() reads for constant while the kernel runs and may move such a load to
// before pdl_wait(), unless it depends on a value that load_in_order() reads behind the wait.  So
// whatever the launch directly before may have written is read with these; __ldg() is for what is older,
// or hangs on a row count read behind the wait.
__device__ __forceinline__ uint32_t load_in_order(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int32_t load_in_order(const int8_t* p) {
  int32_t v;
  asm volatile("ld.global.s8 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int32_t load_in_order(const uint16_t* p) {
  int32_t v;
  asm volatile("ld.global.u16 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t st, Args&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace spconvb
