/* Preloaded in front of the CUDA runtime: answers cooperative launches the way it does where a grid does not fit at once into the SMs that the process may use. */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <stdio.h>

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *config, const void *kernel, void **args) {
    for (unsigned i = 0; i < config->numAttrs; ++i)
        if (config->attrs[i].id == cudaLaunchAttributeCooperative && config->attrs[i].val.cooperative) {
            fputs("refused\n", stderr);
            return cudaErrorCooperativeLaunchTooLarge;
        }
    cudaError_t (*launch)(const cudaLaunchConfig_t *, const void *, void **) = dlsym(dlopen("libcudart.so.12", RTLD_NOW | RTLD_NOLOAD), "cudaLaunchKernelExC");
    return launch(config, kernel, args);
}
