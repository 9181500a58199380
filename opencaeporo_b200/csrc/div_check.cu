// div_check.cu -- the kernels' own divisions (flash_div.cuh, div_const in
// flash_common.cuh) on arrays, so that they can be compared with `/`.
#include "flash_common.cuh"
#include "flash_div.cuh"
#include "ocp_flash.h"

namespace ocpf {

__global__ void __launch_bounds__(256) k_check_division(int form, int64_t n, const double* a, const double* b, double* q)
{
    for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const double x = a[i], y = b[i];
        double       v = 0;
        switch (form) {
            case 0: v = x / y; break;
            case 1: v = div1(x, y); break;
            case 2: v = div_core(x, y); break;
            case 3: v = div_const(x, 3, RCP3); break;
            case 4: v = div_const(x, 9, RCP9); break;
            case 5: v = div_const(x, 54, RCP54); break;
            case 6: v = div_const(x, D1MD2, RCPD1MD2); break;
            case 7: v = __fma_rn(-y, div_seed(y), 1.0); break;
        }
        q[i] = v;
    }
}

}  // namespace ocpf

extern "C" int ocpf_check_division(int form, int64_t n, const double* a, const double* b, double* q, void* stream)
{
    if (form < 0 || form > 7 || n < 0 || (n > 0 && (!a || !b || !q))) return OCPF_EINVAL;
    if (n == 0) return OCPF_OK;
    const int64_t blocks = (n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096;
    ocpf::k_check_division<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(form, n, a, b, q);
    return cudaGetLastError() == cudaSuccess ? OCPF_OK : OCPF_ECUDA;
}
