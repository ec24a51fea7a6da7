// Host build of the volumetric kernels' dealing order. Test-only.
#include "../../grrt_b200/csrc/device/vol_steps.cuh"

extern "C" void vol_deal(unsigned total, unsigned lanes, unsigned warps, unsigned* out) {
    for (unsigned k = 0; k < total; ++k) out[k] = grrt_b200::vol_deal_order(k, total, lanes, warps);
}
