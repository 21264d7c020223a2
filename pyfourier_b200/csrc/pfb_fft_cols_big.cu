// Column passes of the stage plans with a radix above 16.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kImageIn, 2>(const ColPass &, cudaStream_t);
template int launch_col_mode<kImageIn, 3>(const ColPass &, cudaStream_t);
template int launch_col_mode<kForward, 2>(const ColPass &, cudaStream_t);
template int launch_col_mode<kForward, 3>(const ColPass &, cudaStream_t);
template int launch_col_mode<kInverse, 2>(const ColPass &, cudaStream_t);
template int launch_col_mode<kInverse, 3>(const ColPass &, cudaStream_t);
template int launch_col_mode<kImageOut, 2>(const ColPass &, cudaStream_t);
template int launch_col_mode<kImageOut, 3>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
