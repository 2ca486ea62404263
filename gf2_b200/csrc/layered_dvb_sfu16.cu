// gf2cuda layered-schedule DVB-T2 kernels: sum-product on the SFU (GF2C_ALGO_SPA_FAST), FP16 messages.
#include "layered_dvb.cuh"

namespace gf2c {

const void* layered_dvb_sfu16_kernel(int D, bool shared_app, int threads) { return dvb_t<L_SPA_FAST, 1>(D, shared_app, threads); }

}  // namespace gf2c
