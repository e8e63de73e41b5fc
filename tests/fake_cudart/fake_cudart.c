/* The CUDA runtime calls that the library's sort makes, answered on the host and preloaded
 * before the real runtime: device memory is host memory, kernels do not run, and a call
 * chosen by the test (fake_fail) returns an error in place of the real one. */
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
int cudaMalloc(void **p, size_t bytes) { return (*p = malloc(bytes)) ? kOk : 2; }
int cudaFree(void *p)
{
    free(p);
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
