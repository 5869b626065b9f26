// smem_emul.cpp -- SmemLimit against a fake CUDA runtime of several devices:
// prints "<name> <count>" per check.
#include <cstdio>

#include "smem_limit.cuh"

static int g_dev, g_set[128], g_fail;

extern "C" cudaError_t cudaGetDevice(int* d)
{
    *d = g_dev;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int)
{
    if (g_fail) return cudaErrorInvalidValue;
    g_set[g_dev]++;
    return cudaSuccess;
}

static void kern(int) {}

int main()
{
    static atmwfs::SmemLimit limit;
    int errors = 0;
    g_fail = 1;
    g_dev = 3;
    errors += limit.raise(kern, 100000) == cudaSuccess;  // a failure is reported and not recorded
    g_fail = 0;
    for (int round = 0; round < 3; round++)
        for (g_dev = 0; g_dev < 70; g_dev++) errors += limit.raise(kern, 100000) != cudaSuccess;
    int once = 0, again = 0;
    for (int d = 0; d < 64; d++) once += g_set[d] == 1;
    for (int d = 64; d < 70; d++) again += g_set[d] == 3;
    printf("errors %d\nonce %d\nagain %d\n", errors, once, again);
    return 0;
}
