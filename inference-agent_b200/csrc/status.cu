// Error reporting and build information of the library, shared by every entry point.
#include <cuda.h>

#include <cstdlib>

#include "ingot_internal.cuh"

static thread_local std::string g_last_error;

void ingot_set_error(const std::string& msg) { g_last_error = msg; }

int ingot_cuda_fail(cudaError_t e, const char* what) {
    g_last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? INGOT_ERR_NOMEM : INGOT_ERR_CUDA;
}

bool ingot_use_pdl() {
    static const bool v = getenv("INGOT_NO_PDL") == nullptr;
    return v;
}

typedef CUresult (*PointerAttributesFn)(unsigned, CUpointer_attribute*, void**, CUdeviceptr);
static PointerAttributesFn pointer_attributes_fn() {
    static const PointerAttributesFn fn = [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult found;
        const bool ok = cudaGetDriverEntryPoint("cuPointerGetAttributes", &sym, cudaEnableDefault, &found) == cudaSuccess && found == cudaDriverEntryPointSuccess;
        return reinterpret_cast<PointerAttributesFn>(ok ? sym : nullptr);
    }();
    return fn;
}

extern "C" {

void* ingot_device_view(const void* host, size_t bytes) {
    unsigned type = 0, managed = 0;
    void* at = nullptr;
    unsigned long long first = 0;
    size_t size = 0;
    CUpointer_attribute which[5] = {CU_POINTER_ATTRIBUTE_MEMORY_TYPE, CU_POINTER_ATTRIBUTE_IS_MANAGED, CU_POINTER_ATTRIBUTE_DEVICE_POINTER, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR,
                                    CU_POINTER_ATTRIBUTE_RANGE_SIZE};
    void* into[5] = {&type, &managed, &at, &first, &size};
    const PointerAttributesFn ask = pointer_attributes_fn();
    // the driver answers for the thread's context, and the runtime binds one only when a call of its own needs it
    static thread_local const bool bound = [] {
        int device = 0;
        const bool ok = cudaGetDevice(&device) == cudaSuccess && cudaSetDevice(device) == cudaSuccess;
        if (!ok) cudaGetLastError();
        return ok;
    }();
    if (!ask || !bound || ask(5, which, into, reinterpret_cast<CUdeviceptr>(host)) != CUDA_SUCCESS || type != CU_MEMORYTYPE_HOST || managed || !at) return nullptr;
    const unsigned long long view = reinterpret_cast<unsigned long long>(at);
    return view >= first && bytes <= size && view - first <= size - bytes ? at : nullptr;
}

const char* ingot_status_string(int status) {
    switch (status) {
        case INGOT_OK: return "ok";
        case INGOT_ERR_INVALID: return "invalid argument";
        case INGOT_ERR_CUDA: return "CUDA call failed";
        case INGOT_ERR_UNSUPPORTED: return "unsupported shape or dtype";
        case INGOT_ERR_NOMEM: return "out of device memory";
        case INGOT_ERR_DEVICE: return "a kernel reported an error";
        default: return "unknown status";
    }
}

const char* ingot_last_error(void) { return g_last_error.c_str(); }

const char* ingot_build_arch(void) { return "sm_100a"; }

const char* ingot_build_flags(void) {
#ifdef INGOT_BOUNDS_CHECK
    return "bounds-check";
#else
    return "";
#endif
}

}  // extern "C"
