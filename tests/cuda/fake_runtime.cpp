// A stand-in for the CUDA runtime under the renderer's host code: device memory is host memory, and a
// launch is only noted, except that the rasteriser leaves marks in the depth buffer and the queue and
// the resolving kernel takes them away, as the kernels do.  Launch `fake_fail_launch` (counted from 0)
// fails, and nothing runs while fake_capturing is set.  fake_dirty_frames counts frames that began on
// buffers another frame had left marks in.
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Dim3 {
    unsigned x, y, z;
};
std::map<const void*, std::string>& names() {  // filled before this file's objects are made
    static std::map<const void*, std::string> m;
    return m;
}
std::vector<std::pair<unsigned char*, size_t>> allocated;  // the depth buffer, then the queue
int last_error = 0, launches = 0, memsets = 0;

int set(void* p, int v, size_t n) {
    std::memset(p, v, n);
    ++memsets;
    return 0;
}

bool marked() {
    for (size_t k = 0; k < allocated[0].second; ++k)
        if (allocated[0].first[k] != 0xFF) return true;
    unsigned long long counts[2];  // of the queue's parts
    std::memcpy(counts, allocated[1].first, sizeof(counts));
    return counts[0] != 0 || counts[1] != 0;
}
}  // namespace

extern "C" {

int fake_fail_launch = -1, fake_dirty_frames = 0, fake_capturing = 0;
int fake_launches() { return launches; }
int fake_memsets() { return memsets; }
void fake_reset() {  // before a renderer is created
    allocated.clear();
    fake_fail_launch = -1;
    fake_dirty_frames = fake_capturing = launches = memsets = 0;
}

static int launch(const void* func) {
    if (launches++ == fake_fail_launch) return last_error = 719;
    if (fake_capturing) return 0;
    const std::string& name = names()[func];
    const unsigned long long one[2] = {1, 1};
    if (name.find("k_splat_raster") != std::string::npos) {
        if (marked()) ++fake_dirty_frames;
        std::memset(allocated[0].first, 0x11, allocated[0].second);
        std::memcpy(allocated[1].first, one, sizeof(one));
    } else if (name.find("k_splat_resolve") != std::string::npos) {
        std::memset(allocated[0].first, 0xFF, allocated[0].second);
        std::memset(allocated[1].first, 0, sizeof(one));
    }
    return 0;
}

void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*,
                            void*, int*) {
    names()[host] = name;
}
unsigned __cudaPushCallConfiguration(Dim3, Dim3, size_t, void*) { return 0; }
int __cudaPopCallConfiguration(Dim3*, Dim3*, size_t*, void**) { return 0; }
int __cudaGetKernel(const void** kernel, const void* func) {
    *kernel = func;
    return 0;
}
int __cudaLaunchKernel(const void* kernel, Dim3, Dim3, void**, size_t, void*) { return launch(kernel); }
int cudaLaunchKernelExC(const void*, const void* func, void**) { return launch(func); }

int cudaMalloc(void** p, size_t n) {
    *p = std::malloc(n);
    allocated.emplace_back(static_cast<unsigned char*>(*p), n);
    return 0;
}
int cudaFree(void*) { return 0; }
int cudaMemset(void* p, int v, size_t n) { return set(p, v, n); }
int cudaMemsetAsync(void* p, int v, size_t n, void*) { return fake_capturing ? 0 : set(p, v, n); }
int cudaStreamSynchronize(void*) { return 0; }
int cudaStreamIsCapturing(void*, int* status) {
    *status = fake_capturing;
    return 0;
}
int cudaDeviceSynchronize() { return 0; }
int cudaGetDevice(int* d) {
    *d = 0;
    return 0;
}
int cudaDeviceGetAttribute(int* v, int, int) {
    *v = 152;
    return 0;
}
int cudaGetLastError() {
    const int e = last_error;
    last_error = 0;
    return e;
}

}  // extern "C"
