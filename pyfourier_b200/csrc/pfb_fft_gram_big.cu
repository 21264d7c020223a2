// The Gram's middle pass of the stage plans with a radix above 16.
#include "pfb_fft_gram.cuh"

namespace pfb {
namespace fft {

template int launch_gram_rows_t<2>(const GramRows &, cudaStream_t);
template int launch_gram_rows_t<3>(const GramRows &, cudaStream_t);

}  // namespace fft
}  // namespace pfb
