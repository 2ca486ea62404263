// gf2cuda layered-schedule DVB-T2 kernels: normalised / offset min-sum (and min-sum), FP16 messages.
#include "layered_dvb.cuh"

namespace gf2c {

const void* layered_dvb_nms16_kernel(int D, bool shared_app, int threads) { return dvb_t<L_NMS, 1>(D, shared_app, threads); }

}  // namespace gf2c
