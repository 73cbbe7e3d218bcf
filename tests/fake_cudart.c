/* A CUDA runtime for tests of host code without a GPU: one device, memory from the heap, kernels that do nothing.  Loaded before
 * the real one (LD_PRELOAD), it counts what is alive and notes the order of copies, synchronisations and launches. */
#include <cuda_runtime_api.h>
#include <stdatomic.h>
#include <stdlib.h>
#include <string.h>
#include <unistd.h>

static atomic_int live, streams, copies_fail, unsynced;   /* unsynced: copies issued and not waited for */

int fake_live(void) { return live; }             /* allocations, streams and events that exist */
int fake_streams_made(void) { return streams; }
int fake_unsynced(void) { return unsynced; }
void fake_fail_copies(int k) { copies_fail = k; }    /* the next k copies return an error */

static cudaError_t take(void** p, size_t n) {
    *p = calloc(1, n ? n : 1);
    live++;
    return cudaSuccess;
}
static cudaError_t drop(void* p) {
    if (p) live--;
    free(p);
    return cudaSuccess;
}
static cudaError_t copy(void* d, const void* s, size_t n) {
    if (copies_fail > 0) { copies_fail--; return cudaErrorUnknown; }
    memcpy(d, s, n);
    unsynced++;
    return cudaSuccess;
}
static cudaError_t handle(void** p) {
    usleep(20000);      /* long enough for a second thread to come in */
    return take(p, 16);
}

/* Launches: no kernel runs; launch i finds the given words in its accumulators. */
enum { LAUNCHES = 4, WORDS = 32 };
static unsigned long long words[LAUNCHES][WORDS];
static const void* fns[LAUNCHES];
static atomic_int launches;
void fake_set_word(int launch, int word, unsigned long long v) { words[launch][word] = v; }
int fake_launches(void) { return launches; }
int fake_same_kernel(int i, int j) { return fns[i] == fns[j]; }
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void** args, size_t sh, cudaStream_t st) {
    const int i = launches++;
    if (i >= LAUNCHES) return cudaErrorUnknown;
    memcpy(*(void**)args[1], words[i], sizeof words[i]);      /* (arguments, accumulators) */
    fns[i] = f;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t sh, unsigned fl) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t sh) {
    *n = 2;
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned f) { return take(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void* p) { return drop(p); }
cudaError_t cudaFreeHost(void* p) { return drop(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, enum cudaMemcpyKind k) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind k, cudaStream_t st) { return copy(d, s, n); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { streams++; return handle((void**)s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return drop(s); }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { unsynced = 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { unsynced = 0; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle((void**)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned f) { return handle((void**)e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return drop(e); }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) { *ms = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp* p, int d) {
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 4;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int d) { *v = 4; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = 1 << 26; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return "an error of the fake runtime"; }
const char* cudaGetErrorName(cudaError_t e) { return "fake"; }
