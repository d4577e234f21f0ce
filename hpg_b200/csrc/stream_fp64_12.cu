// stream_fp64_12.cu -- the stream kernel's fp64 form, 1 and 2 polarizations.
#include "stream_launch.cuh"

namespace hpgb {
namespace stream {

template Status launch_stream_n<kFP64, 1>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);
template Status launch_stream_n<kFP64, 2>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);

}  // namespace stream
}  // namespace hpgb
