// gf2cuda layered-schedule decoder (sm_100a): host-side kernel selection.
// The device code is in layered_impl.cuh; the kernels are instantiated in
// layered_{sfu,nms,spa}{16,32}.cu (one translation unit per check-node rule
// and message type, so that they compile in parallel).
#include "internal.h"

namespace gf2c {

enum { L_MS = 0, L_SPA = 1, L_NMS = 2, L_SPA_FAST = 3 };

const void* layered_sfu16_kernel(int dcmax, int maxt, bool stage, int bps);
const void* layered_sfu32_kernel(int dcmax, int maxt, bool stage, int bps);
const void* layered_nms16_kernel(int dcmax, int maxt, bool stage, int bps);
const void* layered_nms32_kernel(int dcmax, int maxt, bool stage, int bps);
const void* layered_spa16_kernel(int dcmax, int maxt, bool stage, int bps);
const void* layered_spa32_kernel(int dcmax, int maxt, bool stage, int bps);

const void* layered_dvb_sfu16_kernel(int D, bool shared_app, int threads);
const void* layered_dvb_sfu32_kernel(int D, bool shared_app, int threads);
const void* layered_dvb_nms16_kernel(int D, bool shared_app, int threads);
const void* layered_dvb_nms32_kernel(int D, bool shared_app, int threads);

int layered_dvb_bucket(const HostCode& h) {
  if (h.kind != 2 || h.z != 360 || h.sp_mode != 1 || !h.layered_ok) return 0;
  const int D = layered_dcmax_bucket(h.max_dc);
  const bool normal = h.n == 64800;
  if (!normal && h.n != 16200) return 0;
  // normal codes: every row group has D slots; short ones: at least as many as
  // the irregular kernels take for granted
  const int least = normal ? D : (D == 7 ? 4 : D == 13 ? 9 : D == 19 ? 16 : D);
  for (const int4& G : h.cg)
    if (G.y != 360 || G.z > D || G.z < least) return 0;
  return D <= 22 ? D : 0;
}

// Layered min-sum runs as normalised / offset min-sum, as below.
const void* layered_dvb_kernel_ptr(int algo, int msg16, int D, bool shared_app, int threads) {
  switch (algo) {
    case L_MS:
    case L_NMS:
      return msg16 ? layered_dvb_nms16_kernel(D, shared_app, threads) : layered_dvb_nms32_kernel(D, shared_app, threads);
    case L_SPA_FAST:
      return msg16 ? layered_dvb_sfu16_kernel(D, shared_app, threads) : layered_dvb_sfu32_kernel(D, shared_app, threads);
  }
  return nullptr;
}

int layered_dcmax_bucket(int max_dc) {
  static const int buckets[] = {7, 9, 10, 11, 13, 14, 18, 19, 22, 26, 32};
  for (int b : buckets)
    if (max_dc <= b) return b;
  return -1;
}

// Layered min-sum runs on the normalised / offset min-sum kernels with
// alpha = 1, beta = 0 (the decoder supplies those weights): 1 * max(m - 0, 0)
// is m exactly, so the messages are bit-identical to plain min-sum.
const void* layered_kernel_ptr(int algo, int msg16, int dcmax, int maxt, bool stage, int bps) {
  switch (algo) {
    case L_MS:
    case L_NMS:
      return msg16 ? layered_nms16_kernel(dcmax, maxt, stage, bps) : layered_nms32_kernel(dcmax, maxt, stage, bps);
    case L_SPA:
      return msg16 ? layered_spa16_kernel(dcmax, maxt, stage, bps) : layered_spa32_kernel(dcmax, maxt, stage, bps);
    case L_SPA_FAST:
      return msg16 ? layered_sfu16_kernel(dcmax, maxt, stage, bps) : layered_sfu32_kernel(dcmax, maxt, stage, bps);
  }
  return nullptr;
}

size_t layered_smem_bytes(int smem_app_floats, int bitmap_words) {
  return (size_t)((bitmap_words * 4 + 15) & ~15) + (size_t)smem_app_floats * 4;
}

}  // namespace gf2c
