// Column passes: the middle of an inverse transform.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kInverse, 0>(const ColPass &, cudaStream_t);
template int launch_col_mode<kInverse, 1>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
