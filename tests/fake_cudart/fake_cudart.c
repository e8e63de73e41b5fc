/* The CUDA runtime calls that the library's sort and the creation of a system make, answered
 * on the host and preloaded before the real runtime: device memory is host memory, kernels
 * do not run, and a call chosen by the test (fake_fail, fake_memory) returns an error in
 * place of the real one. */
#include <stdlib.h>
#include <string.h>

enum { kOk = 0, kInvalidValue = 1, kLaunchOutOfResources = 701 };

static int g_launch_fails = -1;    /* launches until one fails (-1: none does) */
static int g_attribute_fails = 0;
static int g_pending = 0;          /* the runtime's last error */
static int g_waits = 0;

static int raise_error(int e)
{
    g_pending = e;
    return e;
}

void fake_fail(int launch, int attribute, int pending)
{
    g_launch_fails = launch;
    g_attribute_fails = attribute;
    g_pending = pending;
    g_waits = 0;
}
int fake_pending(void) { return g_pending; }
int fake_waits(void) { return g_waits; }

static int launch(void)
{
    if (g_launch_fails == 0) return raise_error(kLaunchOutOfResources);
    if (g_launch_fails > 0) --g_launch_fails;
    return kOk;
}
int cudaLaunchKernelExC(const void *config, const void *kernel, void **args)
{
    (void)config, (void)kernel, (void)args;
    return launch();
}
/* what a launch in angle brackets calls */
int __cudaLaunchKernel() { return launch(); }
int __cudaGetKernel(void **kernel, const void *entry)
{
    *kernel = (void *)entry;
    return kOk;
}
int cudaFuncSetAttribute(const void *kernel, int attribute, int value)
{
    (void)kernel, (void)attribute, (void)value;
    return g_attribute_fails ? raise_error(kInvalidValue) : kOk;
}
int cudaGetLastError(void)
{
    const int e = g_pending;
    g_pending = 0;
    return e;
}
int cudaPeekAtLastError(void) { return g_pending; }
int cudaGetDevice(int *device) { return *device = 0; }
int cudaDeviceGetAttribute(int *value, int attribute, int device)
{
    (void)attribute, (void)device;
    *value = 152;
    return kOk;
}
/* device memory in use, and how much there is (-1: as much as asked for) */
static long long g_used = 0, g_limit = -1;
void fake_memory(long long limit) { g_limit = limit; }
long long fake_used(void) { return g_used; }
int cudaMalloc(void **p, size_t bytes)
{
    long long *block;
    *p = NULL;
    if (g_limit >= 0 && g_used + (long long)bytes > g_limit) return raise_error(2);
    if (!(block = malloc(bytes + 64))) return raise_error(2);
    block[0] = (long long)bytes;
    g_used += (long long)bytes;
    *p = (char *)block + 64;
    return kOk;
}
int cudaFree(void *p)
{
    if (p) {
        long long *block = (long long *)((char *)p - 64);
        g_used -= block[0];
        free(block);
    }
    return kOk;
}
int cudaMemset(void *p, int value, size_t bytes)
{
    memset(p, value, bytes);
    return kOk;
}
int cudaStreamCreateWithFlags(void **stream, unsigned flags)
{
    (void)flags;
    *stream = &g_used;
    return kOk;
}
int cudaStreamDestroy(void *stream)
{
    (void)stream;
    return kOk;
}
int cudaHostAlloc(void **p, size_t bytes, unsigned flags)
{
    (void)flags;
    return cudaMalloc(p, bytes);
}
int cudaHostGetDevicePointer(void **device, void *host, unsigned flags)
{
    (void)flags;
    *device = host;
    return kOk;
}
int cudaMemsetAsync(void *p, int value, size_t bytes, void *stream)
{
    (void)stream;
    memset(p, value, bytes);
    return kOk;
}
int cudaMemcpyAsync(void *to, const void *from, size_t bytes, int kind, void *stream)
{
    (void)kind, (void)stream;
    memcpy(to, from, bytes);
    return kOk;
}
int cudaStreamSynchronize(void *stream)
{
    (void)stream;
    ++g_waits;
    return kOk;
}
/* the fixed scratch of the sort without allocation (20 MB hold it) */
int cudaGetSymbolAddress(void **p, const void *symbol)
{
    static char scratch[20 << 20];
    (void)symbol;
    *p = scratch;
    return kOk;
}
int cudaGetDriverEntryPointByVersion(const char *name, void **p, unsigned version, unsigned long long flags, int *found)
{
    (void)name, (void)version, (void)flags;
    *p = 0;
    *found = 1;
    return kOk;
}
