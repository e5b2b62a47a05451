// vah_kernels.cuh -- kernel launch interface shared by vah_kernels.cu and vah_api.cu.
#pragma once

#include <cuda_runtime.h>

#include "vah_stage.cuh"
#include "vah_validity.cuh"

namespace vah {

// One fused RK stage over all interior cells.
template <typename S>
cudaError_t launch_stage(const StageArgs<S> &a, int physics, cudaStream_t stream);

// ---- flux/cell split -------------------------------------------------------
// A split stage is two launches: the flux differences along every axis (kinds
// kFaceX, kFaceY, kFaceZ, which can also be launched one by one to time them),
// then the cells (kCell). One register cap each, the fastest of its candidates
// on the 121x121x81 event: FP64 fluxes 128 (5 blocks' 96 spill in the marches:
// 152 us against 105 along y), FP64 cells 128 in blocks of 64 threads (0.610 ms
// per stage against 0.620 at 168, although they spill), but 168 in 2+1D, where
// the cell needs less (0.090 ms per stage of a 395x395 event against 0.095), FP32
// cells 96 (0.392 against 0.401 at 80; in blocks of 128 threads 0.408).
enum SplitKind { kFaceX = 0, kFaceY = 1, kFaceZ = 2, kCell = 3, kNumSplitKinds = 4 };
constexpr int kFluxThreads = 128, kCellThreads = 64;
template <typename S>
constexpr int kFluxMinb = sizeof(S) == 8 ? 4 : 5;
template <typename S, bool IS3D>
constexpr int kCellMinb = sizeof(S) == 4 ? 10 : (IS3D ? 8 : 6);

// The stage launches of small FP64 2+1D events follow one another as
// programmatic dependents: a launch's blocks may become resident while the last
// blocks of the one before it still run, and wait there for its end before they
// read anything it or an earlier launch wrote (after_previous_launch, which also
// lets the next launch in). Every stage launch waits, so each one's end implies
// those before it. That takes launch latency and a grid's ramp-up off the
// chain: 45.5 -> 40.5 us per step at 61x61, 63.3 -> 62.1 at 200x200, 171.8 ->
// 163.3 at 401x389. Elsewhere it gains nothing or loses, since cell blocks that
// start beside flux blocks inherit their split of L1 and shared memory: 25x23x9
// 50.4 -> 52.7, 121x121x81 616 -> 679 us per stage, FP32 200x200 55.6 -> 66.2.
constexpr int kDependentCells = 189440;  // 2.5 waves of 16 warps per SM
template <typename S>
bool follows_closely(const StageArgs<S> &a) {
    return sizeof(S) == 8 && a.nz == 1 && (long long)a.nx * a.ny <= kDependentCells;
}
#ifdef __CUDACC__
__device__ __forceinline__ void after_previous_launch() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <typename... P, typename... A>
cudaError_t launch_stage_kernel(void (*kernel)(P...), bool dependent, int grid, int block, size_t smem,
                                cudaStream_t stream, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = dependent;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
#endif

// Cells per march segment along an axis of n cells, from the number of warps
// a segment length makes: the fewest waves (148 SMs x minb blocks x 4 warps)
// times the segment's length plus its start-up (one face and its first
// loads, about 1.5 cells' work). The lengths tried are those of n cells in 1, 2,
// ... parts, each once (fewer than 2 sqrt(n): a batch sums over its events for each).
template <typename Warps>
inline int march_segment(int n, int minb, Warps warps) {
    const long long wave = 148 * 4 * minb;
    int best = 1;
    double cost = 1e300;
    for (int len = n; len >= 1;) {
        const double c = (double)((warps(len) + wave - 1) / wave) * (len + 1.5);
        if (c < cost) {
            cost = c;
            best = len;
        }
        if (len == 1) break;
        const int parts = (n + len - 2) / (len - 1);  // the fewest whose cells are shorter
        len = (n + parts - 1) / parts;
    }
    return best;
}

// One launch of one split kind over the planes from k0 that D holds (a.D must
// point at the difference buffers). exact = the reference's per-cell face
// evaluation (FP64).
template <typename S>
cudaError_t launch_split_kind(const StageArgs<S> &a, int physics, bool exact, int kind, cudaStream_t stream);

// One RK stage on the flux/cell split: the flux launch, then the cell launch.
template <typename S>
cudaError_t launch_stage_split(const StageArgs<S> &a, int physics, bool exact, cudaStream_t stream);

// Validity diagnostics of every interior cell after a step.
template <typename S>
cudaError_t launch_validity(const ValidityArgs<S> &a, int physics, cudaStream_t stream);

// A set of device field pointers, passed to kernels by value.
template <typename S>
struct FieldSet {
    S *f[32];
    int n;
};

// The set-up launches below index cell (i, j, k) of the ghosted grid at
// i + pitch (j + (ny + 4) k): pitch = nx + 4 in the reference layout.
// Primitive -> conserved over the interior (setConservedVariables):
// q = 16 conserved slots, u/up = 4 velocity components each.
template <typename S>
cudaError_t launch_set_conserved(const FieldSet<S> &q, const FieldSet<S> &u, const FieldSet<S> &up, const S *e,
                                 int physics, int nx, int ny, int nz, int pitch, double t, int pl_from_field,
                                 cudaStream_t stream);

// Interior primitives for a fresh event: p = EoS(e), u = (1,0,0,0),
// pi = Pi = 0, P_L = p (q[4]).
template <typename S>
cudaError_t launch_init_primitives(const FieldSet<S> &q, const FieldSet<S> &u, const S *e, S *p, const Eos &eos,
                                   int nx, int ny, int nz, int pitch, cudaStream_t stream);

// Rows [row0, row0 + rows) of a field (of nx or, with ghosts, nx + 4 values;
// numbered along y, then eta) between its device layout and a contiguous FP64
// buffer: what a host read or write moves in one copy.
template <typename S>
cudaError_t launch_pack(const S *field, double *packed, int nx, int ny, int pitch, bool ghosts, long long row0,
                        long long rows, cudaStream_t stream);
template <typename S>
cudaError_t launch_unpack(S *field, const double *packed, int nx, int ny, int pitch, bool ghosts, long long row0,
                          long long rows, cudaStream_t stream);

// A field between host memory and the device through `stage` (stage_values
// FP64 values of device memory), a run of rows at a time in stream order. The
// host side is FP64 in the reference layout (full or interior). One contiguous
// copy per run: a 2-D copy per eta plane took 0.6 ms for an interior field of
// the 121x121x81 event against 0.2, and FP32 fields went through a pageable
// host buffer and a host loop (1.8 ms).
constexpr size_t kFieldStageValues = 1u << 20;  // 8 MB, or the field where that is less
inline size_t field_stage_values(size_t ghosted_values) {
    return ghosted_values < kFieldStageValues ? ghosted_values : kFieldStageValues;
}
template <typename S>
cudaError_t read_field(const S *field, double *host, int nx, int ny, int nz, int pitch, bool ghosts, double *stage,
                       size_t stage_values, cudaStream_t stream) {
    if (ghosts && sizeof(S) == sizeof(double) && pitch == nx + 4)  // the layouts agree
        return cudaMemcpyAsync(host, field, sizeof(double) * pitch * (ny + 4) * (nz + 4), cudaMemcpyDeviceToHost, stream);
    if (!ghosts && sizeof(S) == sizeof(double) && nz == 1)  // one plane is one 2-D copy
        return cudaMemcpy2DAsync(host, sizeof(double) * nx, field + 2 + (size_t)pitch * (2 + 2 * (size_t)(ny + 4)),
                                 sizeof(double) * pitch, sizeof(double) * nx, ny, cudaMemcpyDeviceToHost, stream);
    const long long w = ghosts ? nx + 4 : nx, total = ghosts ? (long long)(ny + 4) * (nz + 4) : (long long)ny * nz;
    const long long run = (long long)(stage_values / w);
    for (long long r = 0; r < total; r += run) {
        const long long rows = total - r < run ? total - r : run;
        cudaError_t e = launch_pack<S>(field, stage, nx, ny, pitch, ghosts, r, rows, stream);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(host + r * w, stage, sizeof(double) * rows * w, cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}
template <typename S>
cudaError_t write_field(S *field, const double *host, int nx, int ny, int nz, int pitch, bool ghosts, double *stage,
                        size_t stage_values, cudaStream_t stream) {
    if (ghosts && sizeof(S) == sizeof(double) && pitch == nx + 4)
        return cudaMemcpyAsync(field, host, sizeof(double) * pitch * (ny + 4) * (nz + 4), cudaMemcpyHostToDevice, stream);
    if (!ghosts && sizeof(S) == sizeof(double) && nz == 1)
        return cudaMemcpy2DAsync(field + 2 + (size_t)pitch * (2 + 2 * (size_t)(ny + 4)), sizeof(double) * pitch, host,
                                 sizeof(double) * nx, sizeof(double) * nx, ny, cudaMemcpyHostToDevice, stream);
    const long long w = ghosts ? nx + 4 : nx, total = ghosts ? (long long)(ny + 4) * (nz + 4) : (long long)ny * nz;
    const long long run = (long long)(stage_values / w);
    for (long long r = 0; r < total; r += run) {
        const long long rows = total - r < run ? total - r : run;
        cudaError_t e = cudaMemcpyAsync(stage, host + r * w, sizeof(double) * rows * w, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = launch_unpack<S>(field, stage, nx, ny, pitch, ghosts, r, rows, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Reference ghost fill, three passes with its loop ranges (setGhostCells).
template <typename S>
cudaError_t launch_ghosts(const FieldSet<S> &fields, int nx, int ny, int nz, int pitch, cudaStream_t stream);
// One pass of it (0: x, 1: y, 2: eta): on 2+1D lattices the eta pass fills the
// eta ghost layers that the steps leave to the reader.
template <typename S>
cudaError_t launch_ghost_pass(const FieldSet<S> &fields, int nx, int ny, int nz, int pitch, int pass,
                              cudaStream_t stream);

}  // namespace vah
