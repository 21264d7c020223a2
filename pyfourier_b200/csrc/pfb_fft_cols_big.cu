// Column passes of the stage plans with a radix above 16.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kImageIn, true>(const ColPass &, cudaStream_t);
template int launch_col_mode<kForward, true>(const ColPass &, cudaStream_t);
template int launch_col_mode<kInverse, true>(const ColPass &, cudaStream_t);
template int launch_col_mode<kImageOut, true>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
