// stream_mixed_34.cu -- the stream kernel's mixed form, 3 and 4 polarizations.
#include "stream_launch.cuh"

namespace hpgb {
namespace stream {

template Status launch_stream_n<kMixed, 3>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);
template Status launch_stream_n<kMixed, 4>(hpgb_gridder*, const StreamPlan&,
                                         const StreamParams&);

}  // namespace stream
}  // namespace hpgb
