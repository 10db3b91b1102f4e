/* Preloaded in front of the CUDA runtime by tests/test_pf32_run_paths_gpu.py:
 * counts the launches that carry a cooperative or a cluster attribute, which
 * in an FP32 filter are the whole-run kernel's, and on request refuses the
 * cooperative ones on the host, as the runtime does when the blocks cannot all
 * be resident. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>

static long watched;
static int refuse;

long launch_watch_count(void) { return watched; }
void launch_watch_refuse(int on) { refuse = on; }

cudaError_t cudaLaunchKernelExC(
    const cudaLaunchConfig_t *config, const void *func, void **args)
{
    static cudaError_t (*real)(
        const cudaLaunchConfig_t *, const void *, void **);
    unsigned i;
    if (real == 0)
        *(void **)&real = dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    for (i = 0; i < config->numAttrs; ++i) {
        const cudaLaunchAttribute *a = config->attrs + i;
        if (a->id != cudaLaunchAttributeCooperative &&
            a->id != cudaLaunchAttributeClusterDimension)
            continue;
        ++watched;
        if (refuse)
            return cudaErrorCooperativeLaunchTooLarge;
    }
    return real(config, func, args);
}
