// Column passes: the middle of an inverse transform.
#include "pfb_fft_cols.cuh"

namespace pfb {
namespace fft {

template int launch_col_mode<kInverse, false>(const ColPass &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
