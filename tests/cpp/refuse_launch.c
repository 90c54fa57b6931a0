/* Preloaded before the CUDA runtime: refuse_launch(k) makes the k-th launch from now on (0: the next one) return an
 * error without being queued, as a launch that the runtime refuses.  Every other launch goes through. */
#define _GNU_SOURCE
#include <dlfcn.h>

typedef int (*launch_fn)(const void* config, const void* function, void** args);

static int countdown = -1;

void
refuse_launch(int k)
{
    countdown = k;
}

int
cudaLaunchKernelExC(const void* config, const void* function, void** args)
{
    static launch_fn launch = 0;
    if (launch == 0)
    {
        launch = (launch_fn)dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
    }
    if (countdown >= 0 && countdown-- == 0)
    {
        return 701; /* cudaErrorLaunchOutOfResources */
    }
    return launch(config, function, args);
}
