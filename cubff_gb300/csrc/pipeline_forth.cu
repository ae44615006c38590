// pipeline_forth.cu — the pipelined kernels of the Forth family.
#include "pipeline_kernel.cuh"

namespace cubff {

PipeKernels forth_pipe_kernels(int lang) {
  switch (lang) {
    case kForth: return pipe_kernels<kForth>();
    case kForthcopy: return pipe_kernels<kForthcopy>();
    case kForthtrivial: return pipe_kernels<kForthtrivial>();
    case kForthtrivialReset: return pipe_kernels<kForthtrivialReset>();
  }
  return {};
}

}  // namespace cubff
