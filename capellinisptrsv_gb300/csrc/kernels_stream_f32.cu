// Explicit instantiation of the stream kernel for VALUE_TYPE float; a translation
// unit of its own, so that the build compiles it beside the other kernels.
#include "kernels_stream.cuh"

namespace capsp {

template cudaError_t launch_stream_solve<float>(const StreamArgs<float> &, bool, bool, int, int, cudaStream_t);
template cudaError_t launch_stream_layout<float>(const StreamBuild<float> &, cudaStream_t);
template cudaError_t launch_stream_values<float>(const StreamBuild<float> &, const int *, const float *, float *, float *, int *,
                                               cudaStream_t);

}  // namespace capsp
