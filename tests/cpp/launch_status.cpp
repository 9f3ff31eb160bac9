// The transforms' launch status, on the CPU: the library's own object file of
// csrc/xform.cu linked with a stand-in for the CUDA runtime, in which a chosen
// launch of a call is refused. Checked for every ring size, direction, tile
// width and for the lifted form: a call whose first or second kernel was
// refused returns that error and leaves none behind, and one whose launches
// succeed returns cudaSuccess. Prints the number of wrong answers.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <initializer_list>

namespace xf { struct Job; }
cudaError_t xf_launch_ntt(const xf::Job*, const xf::Job*, int, int, bool, cudaStream_t);
cudaError_t xf_launch_ntt_lift(const xf::Job*, int, int, cudaStream_t);

static int launches, refuse;
static cudaError_t last = cudaSuccess;
static cudaError_t launch() {
    if (++launches != refuse) return cudaSuccess;
    return last = cudaErrorLaunchOutOfResources;
}

extern "C" {
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return launch(); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return launch(); }
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = dim3{1, 1, 1};
    *b = dim3{1, 1, 1};
    *m = 0;
    *(void**)s = nullptr;
    return cudaSuccess;
}
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
}

int main() {
    int wrong = 0, calls = 0;
    const xf::Job* jobs = reinterpret_cast<const xf::Job*>(64);
    for (int logn = 9; logn <= 16; ++logn)
        for (int njobs : {1, 100000})
            for (int form = 0; form < 3; ++form)
                for (refuse = 0; refuse <= 2; ++refuse) {
                    launches = 0;
                    const cudaError_t e = form == 2 ? xf_launch_ntt_lift(jobs, njobs, logn, nullptr)
                                                    : xf_launch_ntt(jobs, nullptr, njobs, logn, form == 1, nullptr);
                    const cudaError_t want = refuse ? cudaErrorLaunchOutOfResources : cudaSuccess;
                    if (e != want || cudaGetLastError() != cudaSuccess) ++wrong;
                    ++calls;
                }
    std::printf("calls=%d wrong=%d\n", calls, wrong);
    return wrong ? 1 : 0;
}
