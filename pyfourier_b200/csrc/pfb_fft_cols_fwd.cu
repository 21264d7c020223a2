// Column passes: the middle of a forward transform.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kForward, 0>(const ColPass &, cudaStream_t);
template int launch_col_mode<kForward, 1>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
