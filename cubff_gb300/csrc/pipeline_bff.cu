// pipeline_bff.cu — the pipelined kernels of the BFF family.
#include "pipeline_kernel.cuh"

namespace cubff {

PipeKernels bff_pipe_kernels(int lang) {
  switch (lang) {
    case kBff: return pipe_kernels<kBff>();
    case kBffNoheads: return pipe_kernels<kBffNoheads>();
    case kBffNoheads4bit: return pipe_kernels<kBffNoheads4bit>();
    case kBffPerm: return pipe_kernels<kBffPerm>();
    case kBff8: return pipe_kernels<kBff8>();
    case kBff8Noheads: return pipe_kernels<kBff8Noheads>();
    case kBffSelfmove: return pipe_kernels<kBffSelfmove>();
  }
  return {};
}

}  // namespace cubff
