// Passes with a gate whose coefficients are not finite (UO_ODD; sqc_unit.cuh): the kernels of sqc_pass.cuh with
// that case in them, in a translation unit of their own to be compiled beside the ordinary ones.
#include "sqc_pass.cuh"

namespace sqc {

int launch_odd_unit_pass(const PassArgs& a, bool dbl, int sms, cudaStream_t st) { return launch_unit_kernel<true>(a, dbl, sms, st); }

int launch_odd_hash_pass(const PassArgs& a, unsigned long long list_hint, bool dbl, int sms, cudaStream_t st) {
    return launch_hash_kernel<true>(a, list_hint, dbl, sms, st);
}

}  // namespace sqc
