// The Gram's middle pass.
#include "pfb_fft_gram.cuh"

namespace pfb {
namespace fft {

template int launch_gram_rows_t<0>(const GramRows &, cudaStream_t);
template int launch_gram_rows_t<1>(const GramRows &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
