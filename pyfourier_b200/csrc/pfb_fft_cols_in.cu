// Column passes: the image side of a forward transform.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kImageIn, 0>(const ColPass &, cudaStream_t);
template int launch_col_mode<kImageIn, 1>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
