// The tensor-core timeout flag's read-and-clear beside a busy default stream: compiles the library's own source and
// drives takeTcError() directly, since no entry point sets the flag.
#include "agb_denoise.cu"

namespace
{
__global__ void k_busy()
{
    for (int i = 0; i < 100; i++)
        __nanosleep(1000000); // each at most 1 ms (2 ms by the instruction's rounding)
}
} // namespace

// flags[0]: what is read after the flag was set; flags[1]: what the next read sees, with the default stream
// busy all the while.
extern "C" __attribute__((visibility("default"))) int tc_flag_probe(int* flags)
{
    int* dev = nullptr;
    const int one = 1;
    cudaStream_t st;
    cudaError_t e = agb::tcErrorFlag(&dev);
    if (e == cudaSuccess)
        e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess)
        return int(e);
    e = cudaMemcpy(dev, &one, sizeof one, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaDeviceSynchronize();
    if (e == cudaSuccess)
    {
        k_busy<<<1, 1>>>();
        e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = agb::takeTcError(flags, st);
    if (e == cudaSuccess)
        e = agb::takeTcError(flags + 1, st);
    const cudaError_t e2 = cudaDeviceSynchronize();
    cudaStreamDestroy(st);
    return int(e != cudaSuccess ? e : e2);
}
