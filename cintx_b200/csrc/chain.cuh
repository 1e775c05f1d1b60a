// Chains of independent launches: the launches of one chunk on the caller's stream, each allowed to start
// before the one ahead of it is through (programmatic stream serialization).  They are independent of one
// another (disjoint outputs, or sums added atomically), and most fill a fraction of the chip.
//
// A launch that kChainNext marks lets the next one start as soon as all its own blocks have started; the
// first launch of a chain starts when everything earlier on the stream is done, so the later ones need wait
// for nothing themselves.  The end of a launch must still mean the end of all before it, for what
// comes after the chain: a launch that kChainPrev marks has one block more than its work takes, which waits
// until the launch ahead is through and does nothing else.  (A wait at the end of a working block costs
// every kernel two to six registers, of (20|10) its third resident block, and 1.6% of a 40-atom sweep.)
// No other stream is involved: a stream held up by its own earlier work holds up nothing else (side
// streams waiting for an event held up every stream that shared their hardware queues).
#pragma once
#include <cuda_runtime.h>

constexpr int kChainPrev = 1;  // may start before the launch ahead of it is through
constexpr int kChainNext = 2;  // the next launch on the stream is a kChainPrev one

#ifdef __CUDACC__
// At the start of a kernel whose work takes blocks [0, nblocks): whether this block has nothing to do.
__device__ __forceinline__ bool chain_begin(int chain, int nblocks) {
  if (chain & kChainNext) asm volatile("griddepcontrol.launch_dependents;");
  if ((int)blockIdx.x < nblocks) return false;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  return true;
}

// Launches kern(args..., chain, blocks).
namespace cintx {
template <class... P, class... A>
inline cudaError_t chain_launch(void (*kern)(P...), unsigned blocks, int threads, size_t smem, cudaStream_t stream,
                                int chain, const A&... args) {
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(blocks + ((chain & kChainPrev) ? 1 : 0));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = (chain & kChainPrev) ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args..., chain, (int)blocks);
}
}  // namespace cintx
#endif
