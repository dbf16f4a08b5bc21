// Error reporting shared by every entry point of the library.
#include <atomic>
#include <cstdarg>
#include <cstdio>

#include "common.cuh"

static thread_local char g_last_error[512] = "";

void fe_set_error(const char* fmt, ...) {
    va_list args;
    va_start(args, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, args);
    va_end(args);
}

int fe_check_launch(const char* what) {
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) {
        fe_set_error("%s: %s", what, cudaGetErrorString(err));
        return 2;
    }
    return 0;
}

// The number of multiprocessors of the current device: the one place kernels' launch heuristics take it from.
int fe_sm_count() {
    static int cached[64] = {0};
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 1;
    if (cached[device] == 0) {
        int sms = 0;
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) return 1;
        cached[device] = sms;
    }
    return cached[device];
}

extern "C" int fe_device_sm_count() { return fe_sm_count(); }

static int g_pdl = 0;

int fe_pdl_enabled() { return g_pdl; }

// Which kernels may overlap their preamble with the tail of the kernel before them: a set of FE_PDL_* classes
// (0: none).  A file's kernels belong to the class it defines before it includes common.cuh.
extern "C" void fe_set_pdl(int classes) { g_pdl = classes; }

// Kernels that may begin while the kernel before them still runs ask for the same split of an SM's memory into shared memory and
// L1.  An SM changes its split only when it is empty: where a kernel of small blocks set it for little shared memory, one
// block of the next kernel fitted where two should have (gate/up of the 7B shape: 128 us instead of 44, the reason why such
// launches were off).  30 % is enough for two of the largest of them and leaves L1 the rows that a weight-streaming kernel reads
// again and again: 16 decode steps of 8 requests on the 7B shape take 25.2 ms with 20 or 30 %, 26.3 with 50 %, 57 with 100 %.
constexpr int SHARED_CARVEOUT_PERCENT = 30;

void fe_share_carveout(const void* kernel) {
    constexpr int SLOTS = 512;
    static std::atomic<const void*> seen[64][SLOTS];         // the kernels that have been told, by their address
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return;
    size_t at = ((size_t)kernel >> 4) % SLOTS;
    for (int i = 0; i < SLOTS; ++i, at = (at + 1) % SLOTS) {
        const void* have = seen[device][at].load(std::memory_order_relaxed);
        if (have == kernel) return;
        if (have == nullptr) {
            cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, SHARED_CARVEOUT_PERCENT);
            seen[device][at].store(kernel, std::memory_order_relaxed);
            return;
        }
    }
}

extern "C" const char* fe_last_error() { return g_last_error; }

extern "C" int fe_abi_version() { return 1; }
