// Column passes: the image side of an inverse transform.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kImageOut, false>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
