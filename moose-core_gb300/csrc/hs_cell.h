// hs_cell.h -- upload of a CellPlan into device memory (one arena per
// solver) and the host mirror used by field access.
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <string>
#include <vector>

#include "hs_device.cuh"
#include "hs_plan.h"

namespace hsg {

// A bump allocator over one device allocation.
struct Arena {
    char* base = nullptr;
    size_t size = 0, used = 0;
    template <class T>
    T* take(size_t n) {
        size_t off = (used + 255) & ~size_t(255);
        used = off + n * sizeof(T);
        return base ? reinterpret_cast<T*>(base + off) : nullptr;
    }
};

// Lays out (dry run with base == nullptr to size the arena) and uploads one
// cell; fills `dc`.  Static arrays are copied with cudaMemcpyAsync on `st`.
// A batch passes `shared`: device arrays it owns (initVm and SynChan
// constants of all cells contiguous, for one-copy reinit) and rate tables
// shared by the cells that have identical ones.  `spikes`: where the spike
// buffers go, if not into `a` (a drop-in solver's: an allocation of more than
// 1 MiB maps memory of its own, ~70 us; smaller ones share a mapping).
std::vector<double> pairTable(const Table& t);   // rate table as the FP64 kernels read it (DevCell::vTab)
struct CellShared {
    double* initVm = nullptr;
    double* synConst = nullptr;
    const double* vTab = nullptr;
    const double* caTab = nullptr;
    const double* g2dBase = nullptr;
    std::vector<uint64_t> g2dOff;    // per gate2d of the cell, offset from g2dBase
};
// `sent`: host copies made on the way, which the caller keeps until it has
// waited for `st` (a copy from pageable memory may be under way when its call
// returns); `programs`: the cell's sweeps, from the dry run to the upload, or
// null to work them out again.
struct CellUpload {
    std::vector<std::shared_ptr<void>> sent;
    std::shared_ptr<void> programs;
};
cudaError_t layoutCell(const CellPlan& P, Arena& a, DevCell& dc, uint32_t spikeCap,
                       cudaStream_t st, CellUpload& up, const CellShared* shared = nullptr, Arena* spikes = nullptr);

// SynChan reinit constants of one cell at the clock dt, 5 per SynChan
// (xc1, xc2, yc1, yc2, norm), computed with the host libm as the reference does.
void synConsts(const CellPlan& P, double dt, double* out);

cudaError_t launchStepFp64(const DevCell& c, uint32_t nsteps, cudaStream_t st);
cudaError_t launchStepFp64Cluster(const DevCell& c, uint32_t ctas, uint32_t nsteps, cudaStream_t st);
uint32_t fp64MatrixRoom();      // doubles of shared memory a drop-in CTA has for its matrix
cudaError_t launchGroupStepFp64(const DevCell* cells, uint32_t n, uint32_t ctas, uint32_t words, uint32_t nsteps,
                                cudaStream_t st);
// The queued field writes of a drop-in solver, one thread each (distinct
// addresses).
cudaError_t launchScatterFields(const FieldWrite* w, uint32_t n, cudaStream_t st);
// HSolveActive::reinit + tick-1/4 object reinit of `nCells` cells, on device.
cudaError_t launchReinitFp64(const DevCell* cells, uint32_t nCells, cudaStream_t st);
// Spike read-back of a batch: per-cell counts (FP64 batch), then the stored
// spikes of every cell gathered at off[c] .. off[c+1] (FP64: from `cells`;
// mixed: `cells` null, from the [cell][cap] arrays srcGen/srcTime).
// out[k] = *src[k] for a gather list of n device addresses (doubles, or
// floats when f32); NaN where src[k] is null.
cudaError_t launchGatherValues(const void* const* src, uint32_t f32, uint64_t n, double* out, cudaStream_t st);
cudaError_t launchSpikeCountsFp64(const DevCell* cells, uint32_t nCells, uint32_t* counts, cudaStream_t st);
cudaError_t launchGatherSpikes(const DevCell* cells, const uint32_t* srcGen, const float* srcTime, uint32_t cap,
                               uint32_t nCells, const uint32_t* off, uint32_t* gen, double* time,
                               cudaStream_t st);
constexpr uint32_t kBatchThreads = 512;     // most threads of the FP64 batch's CTA (128 registers each)
uint32_t fp64BatchWords(uint32_t teams);    // doubles of shared memory it has for matrices
cudaError_t launchBatchStepFp64(const DevCell* cells, const uint32_t* wholePtr, const uint32_t* wholeCells,
                                const uint32_t* teamPtr, const uint32_t* teamCells, uint32_t nBlocks,
                                uint32_t teams, uint32_t teamThreads, uint32_t words, uint32_t nsteps,
                                cudaStream_t st);

}  // namespace hsg
