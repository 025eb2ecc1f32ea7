// Register-gather forward kernel instantiations, BF16 X.
#include "launch.cuh"

namespace cbm {
template <int FORM>
int launch_form(cbm_plan* P, const FwdArgs& a, int32_t ydt, bool vec, int vpl, cudaStream_t st) {
  if (ydt == CBM_F32) {
    return vec ? launch_fwd_v<__nv_bfloat16, float, 8, FORM>(P, a, vpl, st)
               : launch_fwd_v<__nv_bfloat16, float, 1, FORM>(P, a, vpl, st);
  }
  return vec ? launch_fwd_v<__nv_bfloat16, __nv_bfloat16, 8, FORM>(P, a, vpl, st)
             : launch_fwd_v<__nv_bfloat16, __nv_bfloat16, 1, FORM>(P, a, vpl, st);
}

int launch_fwd_bf16(cbm_plan* P, const FwdArgs& a, int32_t ydt, bool vec, int vpl, cudaStream_t st) {
  return a.gin ? launch_form<FORM_GIN>(P, a, ydt, vec, vpl, st) : launch_form<FORM_PLAIN>(P, a, ydt, vec, vpl, st);
}
}  // namespace cbm
