/*
 * fake_cuda.c -- TEST INFRASTRUCTURE: failing CUDA runtime calls, preloaded
 * into a process of its own (tests/fakes.py) so that a library's handling of
 * the failure can be tested on the host.  Nothing fails until armed; a
 * refusal is the runtime's own, of a request that cannot be met (an
 * allocation of 2^60 bytes, a cooperative grid that cannot be resident).
 */
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <string.h>

int fake_malloc_at = -1;  /* the n-th cudaMalloc from now is refused (once) */
int fake_launch_at = -1;  /* the n-th cooperative launch from now is refused (once); -2: all */
int fake_read4 = 0;       /* 4-byte asynchronous reads return 1 */
int fake_launches = 0;    /* cooperative launches asked for */
int fake_cut_at = -1;     /* the n-th cooperative launch from now, one of sdtw::k_steps (Dev, t0, t1, epoch0, taped,
                           * words), runs the first half of its steps and leaves word 7 as after a barrier that gave
                           * up (once) */

cudaError_t cudaMalloc(void** p, size_t bytes)
{
    static cudaError_t (*real)(void**, size_t);
    if (!real)
        real = (cudaError_t(*)(void**, size_t))dlsym(RTLD_NEXT, "cudaMalloc");
    if (fake_malloc_at >= 0 && fake_malloc_at-- == 0)
        bytes = (size_t)1 << 60;
    return real(p, bytes);
}

cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3 block, void** args, size_t smem,
                                        cudaStream_t st)
{
    static cudaError_t (*real)(const void*, dim3, dim3, void**, size_t, cudaStream_t);
    if (!real)
        real = (cudaError_t(*)(const void*, dim3, dim3, void**, size_t, cudaStream_t))dlsym(
            RTLD_NEXT, "cudaLaunchCooperativeKernel");
    fake_launches++;
    if (fake_launch_at == -2 || (fake_launch_at >= 0 && fake_launch_at-- == 0))
        grid.x *= 1024;
    if (fake_cut_at >= 0 && fake_cut_at-- == 0) {
        const int t0 = *(int*)args[1], t1 = *(int*)args[2];
        int half = (t0 + t1) / 2;
        void* cut[6] = {args[0], args[1], &half, args[3], args[4], args[5]};
        cudaError_t e = real(f, grid, block, cut, smem, st);
        cudaMemsetAsync(*(char**)args[5] + 8 * 16 * 7, 1, 8, st);
        return e;
    }
    return real(f, grid, block, args, smem, st);
}

cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, enum cudaMemcpyKind kind, cudaStream_t st)
{
    static cudaError_t (*real)(void*, const void*, size_t, enum cudaMemcpyKind, cudaStream_t);
    if (!real)
        real = (cudaError_t(*)(void*, const void*, size_t, enum cudaMemcpyKind, cudaStream_t))dlsym(
            RTLD_NEXT, "cudaMemcpyAsync");
    if (fake_read4 && n == 4 && kind == cudaMemcpyDeviceToHost) {
        const int one = 1;
        memcpy(dst, &one, 4);
        return cudaSuccess;
    }
    return real(dst, src, n, kind, st);
}
