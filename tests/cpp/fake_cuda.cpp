// A stand-in for the CUDA runtime and the kernel launches, for tests of the
// host code (hs_api.cpp, hs_batch_api.cpp, hs_cell.cu) without a GPU
// (tests/fake_gpu.py).  Device memory is host memory and all streams are one
// queue.  What CUDA leaves open is taken at its worst: a copy between device
// and pageable host memory, which "might be synchronous", reads and writes the
// host's memory only when something waits for it (fake_lazy).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>

#include "hs_cell.h"
#include "hs_mixed.cuh"
#include "hs_noalloc.h"
#include "hs_shared.h"

namespace {

std::deque<std::function<void()>> g_queue;
bool g_lazyRead = false, g_lazyWrite = false;      // device to host, host to device
void drain() {
    while (!g_queue.empty()) {
        g_queue.front()();
        g_queue.pop_front();
    }
}
cudaError_t push(std::function<void()> f) {
    g_queue.push_back(std::move(f));
    return cudaSuccess;
}
std::map<void*, std::pair<int, size_t>> g_made;      // device allocations: number, bytes
int g_count = 0;
void* grab(size_t n) { return std::aligned_alloc(256, (n + 255) / 256 * 256); }
void drop(void* p) {
    g_made.erase(p);
    std::free(p);
}

int g_queries = 0, g_waits = 0;     // calls of cudaEventQuery and cudaStreamWaitEvent
uint32_t g_elimWarps = 0;           // of the last mixed step: of a pair's, else a global, else a shared forest
uint32_t g_teams = 0, g_teamThreads = 0;      // of the last FP64 batch step
int g_device = 0;
std::map<std::pair<int, const void*>, int> g_limit;      // dynamic shared memory each kernel may take, per device
const hsg::DevCell* g_cells = nullptr;      // of the last reinit
uint32_t g_nCells = 0;

constexpr int kShared = 232448, kSharedSm = 233472, kSms = 152;

}  // namespace

extern "C" {

void fake_lazy(int reads, int writes) {
    drain();
    g_lazyRead = reads;
    g_lazyWrite = writes;
}

// Digest of the device allocations made since the last call, in order, but for
// those of `skip` bytes (the cells' descriptions, which hold addresses).
uint64_t fake_digest(uint64_t skip) {
    drain();
    static int from = 0;
    std::map<int, std::pair<const unsigned char*, size_t>> order;
    for (const auto& m : g_made)
        if (m.second.first >= from && m.second.second != skip)
            order[m.second.first] = {static_cast<const unsigned char*>(m.first), m.second.second};
    from = g_count;
    uint64_t h = 1469598103934665603ull;
    for (const auto& o : order)
        for (size_t i = 0; i < o.second.second; ++i) h = (h ^ o.second.first[i]) * 1099511628211ull;
    return h;
}
uint64_t fake_cell_bytes() { return sizeof(hsg::DevCell); }

// Cell k's rate table on Vm as the last reinit had it: {columns, rows} and its data.
const double* fake_table(uint32_t k, uint32_t* shape) {
    drain();
    if (k >= g_nCells) return nullptr;
    shape[0] = g_cells[k].vCol;
    shape[1] = g_cells[k].vRows;
    return g_cells[k].vTab;
}

void fake_teams(uint32_t* n, uint32_t* threads) {
    *n = g_teams;
    *threads = g_teamThreads;
}
uint32_t fake_elim_warps() { return g_elimWarps; }
int fake_queries() { return g_queries; }
int fake_waits() { return g_waits; }

// Whether cell k of the last reinit has a program for its forward sweep.
int fake_has_forward(uint32_t k) {
    drain();
    if (k >= g_nCells) return -1;
    const hsg::DevCell& c = g_cells[k];
    return c.fWaves ? c.fWavePtr && c.fWaveOps : c.fLevelPtr && c.fOpPtr && c.fOps && c.fRun && c.fRunRow;
}

// Readies a kernel for its launches on `device`, and what they may take there.
int fake_allow(uint64_t id, int device) {
    g_device = device;
    const cudaError_t e = hsg::allowShared((const void*)id);
    g_device = 0;
    return e == cudaSuccess ? 0 : -1;
}
int fake_limit(uint64_t id, int device) {
    auto it = g_limit.find({device, (const void*)id});
    return it == g_limit.end() ? 48 * 1024 : it->second;
}

const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {      // kernel `id`: id & 0xFFFF bytes of its own
    *a = {};
    a->sharedSizeBytes = (size_t)f & 0xFFFF;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    if (v + (int)((size_t)f & 0xFFFF) > kShared) return cudaErrorInvalidValue;
    g_limit[{g_device, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? kSms : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kShared : kSharedSm;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t* p, int) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = grab(n);
    std::memset(*p, 0xA5, n);
    g_made[*p] = {g_count++, n};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { drain(); drop(p); return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return push([=] { drop(p); }); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return push([=] { std::memset(p, v, n); }); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    push([=] { std::memcpy(d, s, n); });
    if (!(k == cudaMemcpyDeviceToHost ? g_lazyRead : k == cudaMemcpyHostToDevice && g_lazyWrite)) drain();
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    drain();
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)grab(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { drain(); std::free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { drain(); return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return g_queue.empty() ? cudaSuccess : cudaErrorNotReady; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) {
    ++g_waits;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = nullptr; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)grab(1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) {
    ++g_queries;
    return g_queue.empty() ? cudaSuccess : cudaErrorNotReady;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }

}  // extern "C"

namespace hsg {

// ---- FP64: the steps change nothing ------------------------------------------
uint32_t fp64MatrixRoom() { return (kShared - sizeof(DevCell)) / 8; }
uint32_t fp64BatchWords(uint32_t teams) { return (kShared - teams * sizeof(DevCell)) / 8; }
cudaError_t launchStepFp64(const DevCell&, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchStepFp64Cluster(const DevCell&, uint32_t, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchGroupStepFp64(const DevCell*, uint32_t, uint32_t, uint32_t, uint32_t, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launchBatchStepFp64(const DevCell*, const uint32_t*, const uint32_t*, const uint32_t*, const uint32_t*,
                                uint32_t, uint32_t teams, uint32_t teamThreads, uint32_t, uint32_t, cudaStream_t) {
    g_teams = teams;
    g_teamThreads = teamThreads;
    return cudaSuccess;
}
cudaError_t launchReinitFp64(const DevCell* cells, uint32_t n, cudaStream_t) {
    g_cells = cells;
    g_nCells = n;
    return push([=] {
        for (const DevCell* c = cells; c < cells + n; ++c) {
            std::memcpy(c->V, c->initVm, c->N * 8);
            std::memcpy(c->ca, c->CaBasal, c->P * 8);
        }
    });
}
cudaError_t launchScatterFields(const FieldWrite* w, uint32_t n, cudaStream_t) {
    return push([=] {
        for (uint32_t i = 0; i < n; ++i) std::memcpy(w[i].addr, &w[i].bits, w[i].size);
    });
}
cudaError_t launchGatherValues(const void* const* src, uint32_t f32, uint64_t n, double* out, cudaStream_t) {
    return push([=] {
        for (uint64_t k = 0; k < n; ++k)
            out[k] = f32 ? *static_cast<const float*>(src[k]) : *static_cast<const double*>(src[k]);
    });
}
cudaError_t launchSpikeCountsFp64(const DevCell*, uint32_t, uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchGatherSpikes(const DevCell*, const uint32_t*, const float*, uint32_t, uint32_t, const uint32_t*,
                               uint32_t*, double*, cudaStream_t) {
    return cudaSuccess;
}

// ---- mixed ---------------------------------------------------------------------
cudaError_t launchForestStepMixed(const MixBatch&, const uint32_t*, const uint32_t*, uint32_t, uint32_t, uint32_t,
                                  uint32_t, uint32_t, uint32_t pairWarps, uint32_t elimWarps, uint32_t globalWarps,
                                  uint32_t, uint32_t, uint32_t modes, uint32_t, cudaStream_t) {
    g_elimWarps = pairWarps ? pairWarps : modes == 1u << kRowsShared ? elimWarps : globalWarps;
    return cudaSuccess;
}
cudaError_t launchForestStepMixedCluster(const MixBatch&, const uint32_t*, const uint32_t*, uint32_t, uint32_t,
                                         uint32_t, uint32_t, uint32_t, uint32_t, uint32_t elimWarps, uint32_t,
                                         uint32_t, cudaStream_t) {
    g_elimWarps = elimWarps;
    return cudaSuccess;
}
cudaError_t launchBatchReinitMixed(const MixBatch&, uint32_t, const double*, const float*, const uint32_t*,
                                   cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launchScatterInject(double* const*, uint8_t* const*, const double*, uint32_t, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launchScatterValues(const ValueWrite*, uint32_t, cudaStream_t) { return cudaSuccess; }
std::mutex& injectStaticLock() {
    static std::mutex m;
    return m;
}
InjectWrite* injectStaging() { return nullptr; }
cudaError_t scatterInjectStatic(int, uint32_t, cudaStream_t) { return cudaSuccess; }

}  // namespace hsg
