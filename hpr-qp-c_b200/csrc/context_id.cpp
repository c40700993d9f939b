#include "pool.h"

#include <cuda.h>
#include <cuda_runtime.h>

namespace hpr {

// cuCtxGetId of the current context, reached through the runtime's driver
// entry points so the library links only cudart; false when the driver does
// not offer it.  Any thread may ask, two of them for the first time at once:
// the lookup is the initialisation of a local static, which one thread does
// while the others wait.
bool current_context_id(unsigned long long *id)
{
    struct Driver {
        CUresult (*get_current)(CUcontext *) = nullptr;
        CUresult (*get_id)(CUcontext, unsigned long long *) = nullptr;
        Driver()
        {
            void *f0 = nullptr, *f1 = nullptr;
            cudaDriverEntryPointQueryResult q0, q1;
            if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f0, cudaEnableDefault, &q0) == cudaSuccess &&
                q0 == cudaDriverEntryPointSuccess &&
                cudaGetDriverEntryPoint("cuCtxGetId", &f1, cudaEnableDefault, &q1) == cudaSuccess &&
                q1 == cudaDriverEntryPointSuccess) {
                get_current = (CUresult(*)(CUcontext *))f0;
                get_id = (CUresult(*)(CUcontext, unsigned long long *))f1;
            }
            cudaGetLastError();  // a missing entry point is not an error of this call
        }
    };
    static const Driver driver;
    if (!driver.get_current || !driver.get_id) return false;
    CUcontext ctx = nullptr;
    if (driver.get_current(&ctx) != CUDA_SUCCESS || ctx == nullptr) return false;
    return driver.get_id(ctx, id) == CUDA_SUCCESS;
}

}  // namespace hpr
