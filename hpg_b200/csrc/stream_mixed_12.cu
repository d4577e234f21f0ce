// stream_mixed_12.cu -- the stream kernel's mixed form, 1 and 2 polarizations.
#include "stream_launch.cuh"

namespace hpgb {
namespace stream {

template Status launch_stream_n<kMixed, 1>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);
template Status launch_stream_n<kMixed, 2>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);

}  // namespace stream
}  // namespace hpgb
