// stream_linear_12.cu -- the stream kernel's linear form, 1 and 2 polarizations.
#include "stream_launch.cuh"

namespace hpgb {
namespace stream {

template Status launch_stream_n<kLinear, 1>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);
template Status launch_stream_n<kLinear, 2>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);

}  // namespace stream
}  // namespace hpgb
