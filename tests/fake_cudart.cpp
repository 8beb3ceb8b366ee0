// A stand-in for the CUDA runtime on the host, linked with the library's own objects, for
// tests of its host code without a GPU: what it does when a call of the runtime fails.
// Device memory is host memory, kernels are not run, captured launches are counted; replaying
// a graph of step kernels (two launches a step) advances the time slot that was written last,
// a second a step.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <set>
#include <string>
#include <vector>

namespace {
struct TimeSlot {  // as the library's TimeState
    double totaltime, dt, dtmax, nextoutputtime, endtime, outputtimestep;
    long long nstep, maxsteps;
    int cur, done, status, pad;
};
struct Exec { int steps; };
struct Graph { int launches; };

std::map<std::string, int> calls, fail_at;
std::map<const void*, std::string> names;
std::set<const void*> streams;
std::set<const void*> events;
cudaError_t last = cudaSuccess;
int capturing = 0, captured = 0, live_graphs = 0;
TimeSlot* slot = nullptr;

cudaError_t result(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
// counts the call; the call set by fake_fail fails
bool fails(const std::string& f)
{
    const int n = ++calls[f];
    auto it = fail_at.find(f);
    return it != fail_at.end() && it->second == n;
}
#define FAKE(f) if (fails(#f)) return result(cudaErrorUnknown)
}  // namespace

extern "C" {
// fails the nth further call of a runtime function (0: none any more)
void fake_fail(const char* f, int nth)
{
    calls[f] = 0;
    if (nth) fail_at[f] = nth;
    else fail_at.erase(f);
}
int fake_calls(const char* f) { return calls[f]; }
int fake_live_graphs() { return live_graphs; }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names[f] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static dim3 cg, cb; static size_t cs; static cudaStream_t cst;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st* st) { cg = g; cb = b; cs = s; cst = st; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) { *g = cg; *b = cb; *s = cs; *(cudaStream_t*)st = cst; return cudaSuccess; }

static cudaError_t launch(const void* f, dim3 g)
{
    if (!g.x || !names.count(f)) return result(cudaErrorInvalidConfiguration);
    if (capturing) captured++;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3, void**, size_t, cudaStream_t) { FAKE(cudaLaunchKernel); return launch(f, g); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { FAKE(cudaLaunchKernelExC); return launch(f, c->gridDim); }

cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int)
{
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 0 : 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int* a, int* b) { *a = *b = 0; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = calloc(1, 1 << 16); return cudaSuccess; }

static cudaError_t alloc(void** p, size_t n) { *p = calloc(1, n ? n : 1); return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return alloc(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { FAKE(cudaMallocAsync); return alloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return alloc(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { memset(a, 0, sizeof(*a)); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
    FAKE(cudaMemcpyAsync);
    if (capturing) return cudaSuccess;
    if (k == cudaMemcpyHostToDevice && n == sizeof(TimeSlot)) slot = (TimeSlot*)d;
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { if (!capturing) memset(d, v, n); return cudaSuccess; }

static cudaError_t stream(cudaStream_t* s) { *s = (cudaStream_t)malloc(1); streams.insert(*s); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return stream(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { FAKE(cudaStreamCreateWithPriority); return stream(s); }
cudaError_t cudaStreamGetPriority(cudaStream_t, int* p) { *p = 0; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { streams.erase(s); free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { FAKE(cudaStreamSynchronize); return cudaSuccess; }
static cudaError_t event(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); events.insert(*e); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return event(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { FAKE(cudaEventCreateWithFlags); return event(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { events.erase(e); free(e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) { *t = 1.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t)
{
    FAKE(cudaEventRecord);
    return events.count(e) ? cudaSuccess : result(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t e, unsigned)
{
    FAKE(cudaStreamWaitEvent);
    return events.count(e) ? cudaSuccess : result(cudaErrorInvalidResourceHandle);
}

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode)
{
    FAKE(cudaStreamBeginCapture);
    if (capturing) return result(cudaErrorStreamCaptureUnsupported);
    capturing = 1;
    captured = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g)
{
    if (!capturing) return result(cudaErrorStreamCaptureInvalidated);
    capturing = 0;
    FAKE(cudaStreamEndCapture);
    *g = (cudaGraph_t) new Graph{captured};
    live_graphs++;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; live_graphs--; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long)
{
    FAKE(cudaGraphInstantiate);
    *x = (cudaGraphExec_t) new Exec{((Graph*)g)->launches / 2};
    return cudaSuccess;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaErrorGraphExecUpdateFailure; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete (Exec*)x; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t)
{
    FAKE(cudaGraphLaunch);
    for (int k = 0; slot && k < ((Exec*)x)->steps; k++) {
        if (slot->done || slot->totaltime >= slot->endtime || slot->nstep >= slot->maxsteps) break;
        slot->totaltime += 1.0;
        slot->dt = slot->dtmax = 1.0;
        slot->nstep++;
        slot->cur ^= 1;
    }
    return cudaSuccess;
}
}
