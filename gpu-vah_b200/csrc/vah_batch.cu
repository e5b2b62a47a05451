// vah_batch.cu -- many events, one launch per kernel kind.
//
// A batch holds up to kMaxSlots events of independent grid sizes. Every
// launch of a step covers all events: a block takes an item of a work-list
// (event slot, part of it), largest event first, so events of uneven sizes
// share one launch and the GPU is filled even by many small events.
// The per-event state lives in one device allocation per event (stream-
// ordered, from the batch's memory pool); per-event descriptors (buffer
// pointers, geometry) and clocks (time, u/u_prev parity, step count) live in
// device arrays, so a whole RK2 step -- flux and cell launches of both stages
// plus the clock advance -- is captured once as a CUDA graph and replayed.
// The graph is re-captured only when events are added or removed.
// The flux differences of a stage are scratch that events share. Where it does
// not hold every event's, the events are stepped in groups that it holds, and an
// event that it does not hold in slabs of planes. It takes what the events leave
// of the batch's capacity, up to kScratchBytes, and kScratchBeyond where they leave
// less. One plane's share, without which an event cannot be stepped, is there from
// admission on, so no step fails for want of it.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "vah.h"
#include "vah_ic_device.cuh"
#include "vah_kernels.cuh"
#include "vah_march.cuh"
#include "vah_powf_exc.h"
#include "vah_tile_cell.cuh"

namespace vah {
namespace {

constexpr int kMaxSlots = 4096;
constexpr int kTX = 32, kTY = 4;

template <typename S>
struct SlotDesc {
    int nx, ny, nz, ncx, ncy;
    long long plane;
    double dx, dy, dz, dt, etabar;
    S *q[16], *qS[16], *ep[2][2], *uA[4], *uB[4], *uS[4];
    unsigned char *fallback;  // per ghosted cell: 1 where the latest cell inversion fell back
    unsigned char *hot;       // per ghosted cell: 1 while e > e_freeze (freeze-out crossings)
    double e_freeze;
    unsigned long long *crossings;  // [down, up] during the current step
    unsigned long long *counters;
};

struct SlotClock {
    double t;
    int parity;  // 0: current velocity in uA, previous in uB; 1: swapped
    int active;
    long long steps;
};

// The planes [k0, k1) of an event that one group steps, and where the scratch
// holds their differences: field n of axis d from D + (d N_q + n) stride.
struct Slab {
    int slot, k0, k1;
    long long stride;
    void *D;
};

// One block's piece of work: four strips (from strip i0) of flux_x (kind 0) or
// of flux_march along y or eta (kind 1, 2) over the cells [r0, r1) along it; or
// the interior cells [i0, min(i0 + 128, r1)) of the event (cell lists).
struct WorkItem {
    int slot, slab, kind, i0, r0, r1;
};
constexpr int kCellItem = kTX * kTY;

// The work-lists: fluxes, 2+1D cells, 3+1D cells.
enum { K_FLUX = 0, K_C2 = 1, K_C3 = 2, K_NUM = 3 };

// StageArgs of one slab and stage (the buffer roles of vah_rk2_step), filled by
// 96 threads together (tid 0 to 95).
template <typename S>
__device__ void make_args(StageArgs<S> &a, const SlotDesc<S> &d, const Slab &b, int nq, const SlotClock &c, int stage,
                          const Eos &eos, int tid) {
    const int warp = tid >> 5, n = tid & 31;
    if (warp == 0) {
        if (n < 16) {
            a.qin[n] = stage == 1 ? d.q[n] : d.qS[n];
            a.qout[n] = stage == 1 ? d.qS[n] : d.q[n];
            a.qavg[n] = d.q[n];
            for (int k = 0; k < 3; ++k)  // indexed by ghosted cells: plane k0 is the scratch's first
                a.D[k][n] = n < nq && (k < 2 || d.nz > 1) ? (S *)b.D + (k * nq + n) * b.stride - (b.k0 + 2) * d.plane : nullptr;
        } else if (n < 20) {
            const int m = n - 16;
            S *u = c.parity ? d.uB[m] : d.uA[m], *up = c.parity ? d.uA[m] : d.uB[m];
            a.uin[m] = stage == 1 ? u : d.uS[m];
            a.upin[m] = stage == 1 ? up : u;
            a.guess[m] = u;
            a.uout[m] = stage == 1 ? d.uS[m] : up;
        } else if (n < 31) {
            a.regmap[n - 20] = nullptr;  // validity diagnostics are an event-path option
        }
    } else if (tid == 32) {
        a.nx = d.nx;
        a.ny = d.ny;
        a.nz = d.nz;
        a.k0 = b.k0;
        a.k1 = b.k1;
        a.ncx = d.ncx;
        a.ncy = d.ncy;
        a.plane = d.plane;
        a.stage2 = stage == 2;
        a.zghosts = d.nz > 1;  // 2+1D: the eta ghost layers are filled when a caller reads them
        a.d_planes = 0;
        a.eos = eos;
        a.counters = d.counters;
        a.fallback = d.fallback;
        a.hot = d.hot;
        a.e_freeze = d.e_freeze;
        a.crossings = d.crossings;
        a.ein = d.ep[stage == 1 ? 0 : 1][0];
        a.pin = d.ep[stage == 1 ? 0 : 1][1];
        a.eout = d.ep[stage == 1 ? 1 : 0][0];
        a.pout = d.ep[stage == 1 ? 1 : 0][1];
    } else if (tid == 64) {
        a.dx = d.dx;
        a.dy = d.dy;
        a.dz = d.dz;
        a.dt = d.dt;
        a.etabar = d.etabar;
        a.t_inv = c.t + d.dt;
        a.t_src = stage == 1 ? c.t : c.t + d.dt;
        finish_args(a);
    }
}

// Both stages' arguments of every slab, once per step (block: a slab,
// threadIdx.y: the stage): the stage launches' blocks copy theirs from there.
template <typename S>
__global__ void args_kernel(const SlotDesc<S> *__restrict__ descs, const Slab *__restrict__ slabs, int nq,
                            const SlotClock *__restrict__ clk, const Eos eos, StageArgs<S> *args) {
    const Slab b = slabs[blockIdx.x];
    if (clk[b.slot].active)
        make_args(args[2 * blockIdx.x + threadIdx.y], descs[b.slot], b, nq, clk[b.slot], threadIdx.y + 1, eos, threadIdx.x);
}

// A block's copy of its item's arguments into shared memory; a barrier before use.
template <typename S>
__device__ __forceinline__ void copy_args(StageArgs<S> &sa, const StageArgs<S> *from, int tid) {
    static_assert(sizeof(StageArgs<S>) % 8 == 0, "copied by 8-byte words");
    const double *src = (const double *)from;
    for (int k = tid; k < (int)(sizeof(StageArgs<S>) / 8); k += kTX * kTY) ((double *)&sa)[k] = __ldg(src + k);
}

template <typename S, int PHYS, bool EXACT>
__global__ void __launch_bounds__(kTX *kTY, kFluxMinb<S>)
    batch_flux_kernel(const StageArgs<S> *__restrict__ args, const WorkItem *__restrict__ work, int stage) {
    extern __shared__ __align__(16) unsigned char march_sm[];  // marches: each warp's columns
    __shared__ StageArgs<S> sa;
    __shared__ TablePointers<S> tab;
    const WorkItem it = work[blockIdx.x];
    const StageArgs<S> *from = args + 2 * it.slab + stage - 1;
    const int warp = threadIdx.x / 32, strip = it.i0 + warp;
    copy_args(sa, from, threadIdx.x);
    set_table_pointers<PHYS>(tab, *from, threadIdx.x);
    __syncthreads();
    S *sm = (S *)march_sm + warp * kMarchValues<S, PHYS>;
    if (it.kind == 0) {
        if (strip < flux_x_strips<S>(sa.nx, sa.ny, sa.k1 - sa.k0)) flux_x<PHYS, EXACT>(sa, tab, strip);
    } else if (it.kind == 1) {
        if (strip < march_strips<S>(sa.nx * (sa.k1 - sa.k0))) flux_march<PHYS, 1, EXACT>(sa, tab, strip, it.r0, it.r1, sm);
    } else {
        if (strip < march_strips<S>(sa.nx * sa.ny)) flux_march<PHYS, 2, EXACT>(sa, tab, strip, it.r0, it.r1, sm);
    }
}

template <typename S, int PHYS, bool IS3D>
__global__ void __launch_bounds__(kTX *kTY, kCellMinb<S, IS3D> / 2)
    batch_cell_kernel(const StageArgs<S> *__restrict__ args, const WorkItem *__restrict__ work, int stage) {
    __shared__ StageArgs<S> sa;
    const WorkItem it = work[blockIdx.x];
    copy_args(sa, args + 2 * it.slab + stage - 1, threadIdx.x);
    __syncthreads();
    const int c = it.i0 + threadIdx.x;
    if (c >= it.r1) return;
    const int r = c / sa.nx, i = c - r * sa.nx, k = r / sa.ny, j = r - k * sa.ny;
    if constexpr (sizeof(S) == 4) cell_compute_f32<PHYS, IS3D>(sa, i + 2, j + 2, k + 2);
    else cell_compute<S, PHYS, IS3D, true>(sa, i + 2, j + 2, k + 2);
}

// End of a step: the clock moves on, and the freeze-out surface volume takes
// the step's net crossings (down - up) times tau dx dy deta at the new time.
__global__ void advance_kernel(SlotClock *clk, const double *dts, int nslots, unsigned long long *cross, double *vol,
                               const double *dv) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < nslots && clk[s].active) {
        const double t_new = clk[s].t + dts[s];
        const double net = (double)cross[2 * s] - (double)cross[2 * s + 1];
        if (net != 0.0) vol[s] += t_new * net * dv[s];
        cross[2 * s] = cross[2 * s + 1] = 0;
        clk[s].t = t_new;
        clk[s].parity ^= 1;
        clk[s].steps += 1;
    }
}

// Freeze-out state at admission: 1 where the interior e exceeds e_freeze.
template <typename S>
__global__ void hot_init_kernel(const S *e, unsigned char *hot, double e_freeze, int nx, int ny, int nz, int pitch) {
    const long long n = (long long)nx * ny * nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % nx), j = (int)((c / nx) % ny), k = (int)(c / ((long long)nx * ny));
        const long long s = (i + 2) + (long long)pitch * ((j + 2) + (long long)(ny + 4) * (k + 2));
        hot[s] = (double)e[s] > e_freeze;
    }
}

// Per-slot maximum of e over the interior cells whose latest inversion
// converged (positive doubles order like their bit patterns), for the
// freeze-out test. A cell whose inversion fell back holds e = 0.999 e_prev and
// u = (1,0,0,0) instead of a solution, so it does not count. Order-
// independent, so deterministic.
template <typename S>
__global__ void max_e_kernel(const SlotDesc<S> *__restrict__ descs, const WorkItem *__restrict__ work, int nwork,
                             unsigned long long *maxbits, int cur_ep) {
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = work[w];
        const SlotDesc<S> &d = descs[it.slot];
        const int cell = it.i0 + threadIdx.y * kTX + threadIdx.x;
        double v = 0.0;
        if (cell < it.r1) {
            const int r = cell / d.nx, i = cell - r * d.nx, j = r % d.ny, k = r / d.ny;
            const long long s = (i + 2) + (long long)d.ncx * (j + 2) + d.plane * (k + 2);
            v = (double)d.ep[cur_ep][0][s];
            if (!(v > 0.0) || d.fallback[s]) v = 0.0;
        }
        unsigned long long b = (unsigned long long)__double_as_longlong(v);
        for (int o = 16; o > 0; o >>= 1) {
            unsigned long long x = __shfl_xor_sync(0xffffffffu, b, o);
            b = x > b ? x : b;
        }
        if ((threadIdx.x & 31) == 0) atomicMax(maxbits + it.slot, b);
    }
}

// Per-item partial sums of the event observables (tau T^tt, T^xx - T^yy,
// T^xx + T^yy, e u^t u_T, e u^t) in FP64 over the cells whose latest
// inversion converged (a fallback cell's state is not a solution), one row
// per cell item; the host adds the rows of each slot in a fixed order.
template <typename S, int PHYS>
__global__ void observables_kernel(const SlotDesc<S> *__restrict__ descs, const SlotClock *__restrict__ clk,
                                   const WorkItem *__restrict__ work, int nwork, double *partial) {
    __shared__ double red[5][kTX * kTY / 32];
    const int tid = threadIdx.y * kTX + threadIdx.x;
    for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
        const WorkItem it = work[w];
        const SlotDesc<S> &d = descs[it.slot];
        const SlotClock c = clk[it.slot];
        const int cell = it.i0 + tid;
        double acc[5] = {0, 0, 0, 0, 0};
        const bool in = cell < it.r1;
        const int r = in ? cell / d.nx : 0, i = in ? cell - r * d.nx : 0, j = r % d.ny, k = r / d.ny;
        const long long s = (i + 2) + (long long)d.ncx * (j + 2) + d.plane * (k + 2);
        if (in && !d.fallback[s]) {  // converged cells only
            S *const *u = c.parity ? d.uB : d.uA;
            const double e = (double)d.ep[0][0][s], p = (double)d.ep[0][1][s], pl = (double)d.q[kSlotPL][s];
            const double ut = (double)u[0][s], ux = (double)u[1][s], uy = (double)u[2][s];
            double pt = 0.5 * (e - pl - poly::Rbar0(pl / e) * (e - 3 * p));
            double pixx = 0, piyy = 0;
            if (Phys<PHYS>::PIMUNU) {
                pixx = (double)d.q[9][s];
                piyy = (double)d.q[12][s];
            }
            if (Phys<PHYS>::BULK) pt += 1.5 * (double)d.q[kSlotPi][s];
            const double txx = e * ux * ux + pt * (1 + ux * ux) + pixx;
            const double tyy = e * uy * uy + pt * (1 + uy * uy) + piyy;
            acc[0] = c.t * (double)d.q[0][s] * d.dx * d.dy * d.dz;
            acc[1] = txx - tyy;
            acc[2] = txx + tyy;
            acc[3] = e * ut * sqrt(ux * ux + uy * uy);
            acc[4] = e * ut;
        }
        for (int m = 0; m < 5; ++m)
            for (int o = 16; o > 0; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
        __syncthreads();
        if ((tid & 31) == 0)
            for (int m = 0; m < 5; ++m) red[m][tid >> 5] = acc[m];
        __syncthreads();
        if (tid < 5) {
            double s = 0;
            for (int q = 0; q < kTX * kTY / 32; ++q) s += red[tid][q];
            partial[(size_t)w * 5 + tid] = s;
        }
    }
}

}  // namespace
}  // namespace vah

using vah::SlotClock;
using vah::SlotDesc;
using vah::WorkItem;

struct vah_batch {
    vah_options opt;
    int nq;
    size_t elem;
    cudaStream_t stream;
    bool own_stream;
    cudaMemPool_t pool;
    size_t capacity, used;
    int sms;
    double *d_tab;
    uint32_t *d_exc;
    int nexc;
    void *d_desc;               // SlotDesc<S>[kMaxSlots]
    SlotClock *d_clk;           // [kMaxSlots]
    double *d_dt;               // [kMaxSlots]
    unsigned long long *d_cross;  // [kMaxSlots * 2] freeze-out crossings of the current step (down, up)
    double *d_vol;              // [kMaxSlots] freeze-out surface volume so far, fm^4
    double *d_dv;               // [kMaxSlots] dx dy deta
    std::vector<double> tab;    // host copy of the EoS table (freeze-out energy densities)
    unsigned long long *d_counters;  // [kMaxSlots * 4]
    unsigned long long *d_maxbits;   // [kMaxSlots]
    struct Slot {
        bool used = false;
        vah_lattice lat{};
        vah_hydro hydro{};
        double dt = 0;
        size_t bytes = 0;
        long long admitted = 0;  // the batch's step count at admission: the velocity buffers' parity since
        void *mem = nullptr;
        std::vector<void *> field;  // VAH_F_* -> device array (current roles resolved at query time)
    };
    std::vector<Slot> slots;
    long long steps;                       // queued since the batch was created
    std::vector<unsigned char> desc_host;  // host mirror of the descriptor array
    double *d_fstage;  // staging of the field reads ...
    size_t fstage;     // ... of this many values
    std::vector<WorkItem> lists[vah::K_NUM];  // the work-lists, kept for their memory
    WorkItem *d_work[vah::K_NUM];
    void *d_args;        // StageArgs<S>[cap_args]: both stages' arguments by slab
    size_t cap_args;     // in StageArgs
    char *d_scratch;     // the flux differences of one group of slabs
    size_t cap_scratch;
    vah::Slab *d_slabs;
    size_t cap_slabs;
    int nslabs;
    struct Group {
        int first[vah::K_NUM], count[vah::K_NUM];  // its runs of the work-lists
    };
    std::vector<Group> groups;
    int nwork[vah::K_NUM];
    size_t cap_work[vah::K_NUM];
    double *d_partial;
    size_t cap_partial;
    bool dirty;
    cudaGraphExec_t graph;
    bool has_graph;
    bool timing;
    cudaEvent_t t0, t1;
    double kernel_ms;
    long long kernel_steps;
};

namespace {

int cuda_status(cudaError_t e) {
    if (e == cudaSuccess) return VAH_OK;
    if (e == cudaErrorMemoryAllocation) return VAH_ERR_NOMEM;
    if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return VAH_ERR_NODEVICE;
    return VAH_ERR_CUDA;
}

#define VAH_TRY(call)                                  \
    do {                                               \
        cudaError_t e_ = (call);                       \
        if (e_ != cudaSuccess) return cuda_status(e_); \
    } while (0)

int nq_of(int physics) { return physics == VAH_IDEAL ? 5 : (physics == VAH_PIMUNU ? 15 : 16); }

// Arrays of one event in its allocation: 16 q, 16 qS, 4 e/p, 4 uA, 4 uB,
// 4 uS; then one byte per cell of fallback flags and one of freeze-out state.
constexpr int kArraysPerEvent = 48;

// The most that the scratch of a group's flux differences takes. With 4 GB a
// batch of 256 2+1D events (sides 81 to 201, 5.84 M cells) is one group: as two,
// its FP64 step had twice the launches and their tails (6.10 against 5.98 ms).
constexpr size_t kScratchBytes = (size_t)4 << 30;
// What it may take beyond the capacity where the events leave less: slabs of
// this size (0.7 M FP64 cells) still fill the GPU, those of one plane do not.
constexpr size_t kScratchBeyond = (size_t)256 << 20;

size_t event_bytes(const vah_batch *b, const vah_lattice *lat) {
    const size_t ncell = (size_t)(lat->nx + 4) * (lat->ny + 4) * (lat->nz + 4);
    const size_t per = (ncell * b->elem + 255) / 256 * 256;
    return per * kArraysPerEvent + 2 * ((ncell + 255) / 256 * 256) + 256;
}

// The flux differences of `planes` planes of an event: bytes of one field (which
// interior planes alone have), and of every field and axis.
size_t diff_field_bytes(const vah_batch *b, const vah_lattice &l, int planes) {
    return ((size_t)(l.nx + 4) * (l.ny + 4) * planes * b->elem + 255) / 256 * 256;
}
size_t diff_bytes(const vah_batch *b, const vah_lattice &l, int planes) {
    return diff_field_bytes(b, l, planes) * (l.nz > 1 ? 3 : 2) * b->nq;
}

vah::Eos batch_eos(const vah_batch *b) {
    vah::Eos eos;
    eos.kind = b->opt.eos == VAH_EOS_TABLE ? 1 : 0;
    eos.zeta = b->opt.zeta == VAH_ZETA_CROSSOVER ? 1 : 0;
    eos.tab = b->d_tab;
    eos.exc = b->d_exc;
    eos.nexc = b->nexc;
    return eos;
}

template <typename S>
SlotDesc<S> *desc_host(vah_batch *b, int slot) {
    return (SlotDesc<S> *)b->desc_host.data() + slot;
}

// Energy density at temperature T (fm^-1): the conformal gas e = 13.8997 T^4
// (EquationOfState.cpp:144 inverted) or the table's monotone T(e), bisected
// in ln e.
double energy_at_temperature(const vah_batch *b, double T) {
    if (b->opt.eos != VAH_EOS_TABLE || b->tab.empty()) return 13.8997 * T * T * T * T;
    const int n = (int)b->tab[0];
    const double *Tt = b->tab.data() + VAH_EOS_TABLE_HEADER + n;
    if (T <= Tt[0]) return b->tab[4];
    if (T >= Tt[n - 1]) return b->tab[6];
    int lo = 0, hi = n - 1;
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (Tt[mid] < T) lo = mid;
        else hi = mid;
    }
    const double w = (T - Tt[lo]) / (Tt[hi] - Tt[lo]);
    return std::exp(b->tab[1] + b->tab[3] * (lo + w));
}

template <typename S>
int fill_slot(vah_batch *b, int slot) {
    vah_batch::Slot &sl = b->slots[slot];
    SlotDesc<S> d;
    memset(&d, 0, sizeof(d));
    d.nx = sl.lat.nx;
    d.ny = sl.lat.ny;
    d.nz = sl.lat.nz;
    d.ncx = sl.lat.nx + 4;
    d.ncy = sl.lat.ny + 4;
    d.plane = (long long)d.ncx * d.ncy;
    d.dx = sl.lat.dx;
    d.dy = sl.lat.dy;
    d.dz = sl.lat.dz;
    d.dt = sl.dt;
    d.etabar = sl.hydro.eta_over_s;
    d.counters = b->d_counters + 4 * slot;
    const size_t ncell = (size_t)d.ncx * d.ncy * (sl.lat.nz + 4);
    const size_t per = (ncell * b->elem + 255) / 256 * 256;
    char *base = (char *)sl.mem;
    size_t off = 0;
    auto next = [&]() {
        S *p = (S *)(base + off);
        off += per;
        return p;
    };
    for (int n = 0; n < 16; ++n) d.q[n] = next();
    for (int n = 0; n < 16; ++n) d.qS[n] = next();
    for (int x = 0; x < 2; ++x)
        for (int y = 0; y < 2; ++y) d.ep[x][y] = next();
    for (int m = 0; m < 4; ++m) d.uA[m] = next();
    for (int m = 0; m < 4; ++m) d.uB[m] = next();
    for (int m = 0; m < 4; ++m) d.uS[m] = next();
    d.fallback = (unsigned char *)(base + off);
    d.hot = (unsigned char *)(base + off + (ncell + 255) / 256 * 256);
    d.e_freeze = energy_at_temperature(b, sl.hydro.freezeout_T_GeV / 0.197326938);
    d.crossings = b->d_cross + 2 * slot;
    *desc_host<S>(b, slot) = d;
    VAH_TRY(cudaMemcpyAsync((char *)b->d_desc + sizeof(SlotDesc<S>) * slot, &d, sizeof(d), cudaMemcpyHostToDevice,
                            b->stream));
    return VAH_OK;
}

template <typename T>
int grow(vah_batch *b, T *&p, size_t &cap, size_t n) {  // device memory for n values; contents lost
    if (n <= cap) return VAH_OK;
    if (p) VAH_TRY(cudaFreeAsync(p, b->stream));
    p = nullptr;
    cap = 0;
    VAH_TRY(cudaMallocFromPoolAsync((void **)&p, n * sizeof(T), b->pool, b->stream));
    cap = n;
    return VAH_OK;
}

// Scratch of `want` bytes where the device has them, else of the half and so on
// down to `least`; contents lost. What it frees stays in the batch's pool, so
// that the old size can be had again.
int set_scratch(vah_batch *b, size_t want, size_t least) {
    if (b->d_scratch) VAH_TRY(cudaFreeAsync(b->d_scratch, b->stream));
    b->d_scratch = nullptr;
    b->cap_scratch = 0;
    b->dirty = true;
    for (;; want = std::max(least, want / 2)) {
        const cudaError_t e = cudaMallocFromPoolAsync((void **)&b->d_scratch, want, b->pool, b->stream);
        if (e == cudaSuccess) break;
        cudaGetLastError();  // an allocation that fails leaves nothing else behind
        b->d_scratch = nullptr;
        if (want <= least) return cuda_status(e);
    }
    b->cap_scratch = want;
    return VAH_OK;
}

// The scratch of the batch's events (and of one more, or null): all their
// differences at once; the least that steps them, a plane of each by itself;
// and the most it may take if they leave `free` bytes of the capacity.
struct ScratchBounds {
    size_t all, least, most;
};
ScratchBounds scratch_bounds(const vah_batch *b, const vah_lattice *more, size_t free) {
    ScratchBounds r{0, 0, 0};
    auto add = [&](const vah_lattice &l) {
        r.all += diff_bytes(b, l, l.nz);
        r.least = std::max(r.least, diff_bytes(b, l, 1));
    };
    for (const vah_batch::Slot &sl : b->slots)
        if (sl.used) add(sl.lat);
    if (more) add(*more);
    r.most = std::max(std::max(r.least, kScratchBeyond), std::min(kScratchBytes, free));
    return r;
}

template <typename Item>
void append(std::vector<WorkItem> &list, int n, Item item) {
    const size_t at = list.size();
    list.resize(at + n);
    for (int m = 0; m < n; ++m) list[at + m] = item(m);
}

// The work-lists, groups and scratch of the admitted events.
template <typename S>
int rebuild_work(vah_batch *b) {
    std::vector<WorkItem>(&lists)[vah::K_NUM] = b->lists;
    for (auto &l : lists) l.clear();
    std::vector<int> order;  // largest event first: its items start first, small ones fill the tail
    for (int s = 0; s < (int)b->slots.size(); ++s)
        if (b->slots[s].used) order.push_back(s);
    auto cells = [&](int s) {
        const vah_lattice &l = b->slots[s].lat;
        return (long long)l.nx * l.ny * l.nz;
    };
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cells(x) > cells(y); });
    // the scratch grows to what the events can use of the room they leave (at
    // least by half, so that a set that grows event by event seldom re-allocates)
    const ScratchBounds sb = scratch_bounds(b, nullptr, b->capacity - b->used);
    int rc = VAH_OK;
    if (std::min(sb.all, sb.most) > b->cap_scratch)
        rc = set_scratch(b, std::min(std::max(sb.all, b->cap_scratch + b->cap_scratch / 2), sb.most), sb.least);
    if (rc != VAH_OK) return rc;
    // slabs that the scratch holds (an event, where it does), and groups of them
    std::vector<vah::Slab> slabs;
    std::vector<std::vector<int>> members;
    size_t held = 0;
    for (int s : order) {
        const vah_lattice &l = b->slots[s].lat;
        int planes = l.nz;
        while (planes > 1 && diff_bytes(b, l, planes) > b->cap_scratch)
            planes = std::max(1, std::min(planes - 1, (int)(b->cap_scratch / diff_bytes(b, l, 1))));
        const int n = (l.nz + planes - 1) / planes;
        for (int m = 0; m < n; ++m) {
            const int k0 = (int)((long long)l.nz * m / n), k1 = (int)((long long)l.nz * (m + 1) / n);
            const size_t field = diff_field_bytes(b, l, k1 - k0), bytes = diff_bytes(b, l, k1 - k0);
            if (members.empty() || held + bytes > b->cap_scratch) {
                members.emplace_back();
                held = 0;
            }
            members.back().push_back((int)slabs.size());
            slabs.push_back({s, k0, k1, (long long)(field / sizeof(S)), b->d_scratch + held});
            held += bytes;
        }
    }
    b->groups.clear();
    for (const std::vector<int> &group : members) {
        vah_batch::Group g;
        for (int k = 0; k < vah::K_NUM; ++k) g.first[k] = (int)lists[k].size();
        int seg[3] = {};  // march segments along y and eta, from the whole group's warps
        for (int dir = 1; dir < 3; ++dir) {
            auto along = [&](const vah::Slab &p) { return dir == 1 ? b->slots[p.slot].lat.ny : p.k1 - p.k0; };
            int longest = 1;
            for (int p : group) longest = std::max(longest, along(slabs[p]));
            seg[dir] = vah::march_segment(longest, vah::kFluxMinb<S>, [&](int len) {
                long long w = 0;
                for (int p : group) {
                    const vah_lattice &l = b->slots[slabs[p].slot].lat;
                    if (dir == 2 && l.nz == 1) continue;
                    const long long strips = vah::march_strips<S>(l.nx * (dir == 1 ? slabs[p].k1 - slabs[p].k0 : l.ny));
                    w += (strips + 3) / 4 * 4 * ((along(slabs[p]) + len - 1) / len);
                }
                return w;
            });
        }
        // the marches first (long), then the x strips, which fill the tail
        for (int kind : {2, 1, 0})
            for (int p : group) {
                const vah::Slab &sl = slabs[p];
                const vah_lattice &l = b->slots[sl.slot].lat;
                if (kind == 2 && l.nz == 1) continue;
                const int nk = sl.k1 - sl.k0;
                const int strips = kind == 0 ? vah::flux_x_strips<S>(l.nx, l.ny, nk)
                                             : vah::march_strips<S>(l.nx * (kind == 1 ? nk : l.ny));
                const int at = kind == 2 ? sl.k0 : 0, n = kind == 0 ? 1 : (kind == 1 ? l.ny : sl.k1);
                const int len = kind == 0 ? 1 : seg[kind], quads = (strips + 3) / 4;
                for (int r0 = at; r0 < n; r0 += len)
                    append(lists[vah::K_FLUX], quads, [&](int m) -> WorkItem {
                        return {sl.slot, p, kind, 4 * m, r0, std::min(r0 + len, n)};
                    });
            }
        for (int p : group) {
            const vah::Slab &sl = slabs[p];
            const vah_lattice &l = b->slots[sl.slot].lat;
            const int first = l.nx * l.ny * sl.k0, end = l.nx * l.ny * sl.k1;
            append(lists[l.nz > 1 ? vah::K_C3 : vah::K_C2], (end - first + vah::kCellItem - 1) / vah::kCellItem,
                   [&](int m) -> WorkItem { return {sl.slot, p, 0, first + vah::kCellItem * m, 0, end}; });
        }
        for (int k = 0; k < vah::K_NUM; ++k) g.count[k] = (int)lists[k].size() - g.first[k];
        b->groups.push_back(g);
    }
    b->nslabs = (int)slabs.size();
    if ((rc = grow(b, b->d_slabs, b->cap_slabs, slabs.size())) != VAH_OK) return rc;
    if (b->nslabs)
        VAH_TRY(cudaMemcpyAsync(b->d_slabs, slabs.data(), sizeof(vah::Slab) * slabs.size(), cudaMemcpyHostToDevice,
                                b->stream));
    auto *args = (vah::StageArgs<S> *)b->d_args;
    rc = grow(b, args, b->cap_args, 2 * slabs.size());
    b->d_args = args;
    if (rc != VAH_OK) return rc;
    for (int k = 0; k < vah::K_NUM; ++k) {
        const size_t n = lists[k].size();
        if ((rc = grow(b, b->d_work[k], b->cap_work[k], n)) != VAH_OK) return rc;
        if (n) VAH_TRY(cudaMemcpyAsync(b->d_work[k], lists[k].data(), n * sizeof(WorkItem), cudaMemcpyHostToDevice,
                                       b->stream));
        b->nwork[k] = (int)n;
    }
    const size_t ncells = (size_t)b->nwork[vah::K_C2] + b->nwork[vah::K_C3];
    if ((rc = grow(b, b->d_partial, b->cap_partial, 5 * ncells)) != VAH_OK) return rc;
    // the copies above read host vectors that die here
    VAH_TRY(cudaStreamSynchronize(b->stream));
    return VAH_OK;
}

int rebuild(vah_batch *b) { return b->elem == sizeof(float) ? rebuild_work<float>(b) : rebuild_work<double>(b); }

// A stage of one group: the flux launch (list K_FLUX) or a cell launch.
template <typename S, int PHYS>
cudaError_t launch_list(vah_batch *b, const vah_batch::Group &g, int list, int stage) {
    using namespace vah;
    const StageArgs<S> *args = (const StageArgs<S> *)b->d_args;
    const WorkItem *w = b->d_work[list] + g.first[list];
    const int n = g.count[list], threads = kTX * kTY;
    if (n == 0) return cudaSuccess;
    if (list == K_FLUX) {
        constexpr size_t smem = kTY * kMarchValues<S, PHYS> * sizeof(S);
        auto kernel = batch_flux_kernel<S, PHYS, false>;
        if constexpr (sizeof(S) == 8)
            if (b->opt.flux == VAH_FLUX_PER_CELL) kernel = batch_flux_kernel<S, PHYS, true>;
        static_assert(smem <= 44 * 1024, "with the arguments, within the default shared memory limit");
        kernel<<<n, threads, smem, b->stream>>>(args, w, stage);
    } else if (list == K_C2) {
        batch_cell_kernel<S, PHYS, false><<<n, threads, 0, b->stream>>>(args, w, stage);
    } else {
        batch_cell_kernel<S, PHYS, true><<<n, threads, 0, b->stream>>>(args, w, stage);
    }
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_list_s(vah_batch *b, const vah_batch::Group &g, int list, int stage) {
    switch (b->opt.physics) {
    case VAH_IDEAL: return launch_list<S, 0>(b, g, list, stage);
    case VAH_PIMUNU: return launch_list<S, 1>(b, g, list, stage);
    default: return launch_list<S, 2>(b, g, list, stage);
    }
}

cudaError_t launch_list_any(vah_batch *b, const vah_batch::Group &g, int list, int stage) {
    return b->elem == sizeof(float) ? launch_list_s<float>(b, g, list, stage) : launch_list_s<double>(b, g, list, stage);
}

int launch_args(vah_batch *b) {
    if (b->nslabs == 0) return VAH_OK;
    const dim3 block(96, 2);
    const vah::Eos eos = batch_eos(b);
    if (b->elem == sizeof(float))
        vah::args_kernel<float><<<b->nslabs, block, 0, b->stream>>>((const SlotDesc<float> *)b->d_desc, b->d_slabs, b->nq,
                                                                    b->d_clk, eos, (vah::StageArgs<float> *)b->d_args);
    else
        vah::args_kernel<double><<<b->nslabs, block, 0, b->stream>>>((const SlotDesc<double> *)b->d_desc, b->d_slabs, b->nq,
                                                                     b->d_clk, eos, (vah::StageArgs<double> *)b->d_args);
    VAH_TRY(cudaGetLastError());
    return VAH_OK;
}

int enqueue_step(vah_batch *b) {
    using namespace vah;
    const int rc = launch_args(b);
    if (rc != VAH_OK) return rc;
    for (int stage = 1; stage <= 2; ++stage)
        for (const vah_batch::Group &g : b->groups)
            for (int list = 0; list < K_NUM; ++list) VAH_TRY(launch_list_any(b, g, list, stage));
    advance_kernel<<<(kMaxSlots + 255) / 256, 256, 0, b->stream>>>(b->d_clk, b->d_dt, kMaxSlots, b->d_cross, b->d_vol,
                                                                 b->d_dv);
    VAH_TRY(cudaGetLastError());
    return VAH_OK;
}

int capture_graph(vah_batch *b) {
    if (b->has_graph) {
        cudaGraphExecDestroy(b->graph);
        b->has_graph = false;
    }
    cudaGraph_t g;
    VAH_TRY(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    int rc = enqueue_step(b);
    cudaError_t e = cudaStreamEndCapture(b->stream, &g);
    if (rc != VAH_OK) return rc;
    VAH_TRY(e);
    e = cudaGraphInstantiate(&b->graph, g, 0);
    cudaGraphDestroy(g);
    VAH_TRY(e);
    b->has_graph = true;
    b->dirty = false;
    return VAH_OK;
}

template <typename S>
vah::FieldSet<S> fs(S *const *p, int n) {
    vah::FieldSet<S> f{};
    for (int k = 0; k < n; ++k) f.f[k] = p[k];
    f.n = n;
    return f;
}

// Device-generated initial energy density (vah_batch_add_glauber) into the
// slot's e interior: participants sampled, deposited and normalised on the
// GPU; scratch from the batch's pool, freed in stream order.
template <typename S>
int glauber_slot(vah_batch *b, const SlotDesc<S> &d, const vah_lattice &lat, const vah_glauber &g) {
    if (g.A < 1 || g.A > 256 || !(g.width > 0) || !(g.ws_R > 0) || !(g.ws_a > 0) || !std::isfinite(g.ws_R + g.ws_a) ||
        (lat.nz > 1 && !(g.sigma_eta > 0)))
        return VAH_ERR_ARG;
    const size_t nxy = (size_t)lat.nx * lat.ny;
    const size_t bytes = 256 + sizeof(double) * (4 * (size_t)g.A + nxy);
    char *scratch = nullptr;
    VAH_TRY(cudaMallocFromPoolAsync((void **)&scratch, bytes, b->pool, b->stream));
    unsigned long long *maxbits = (unsigned long long *)scratch;
    int *d_np = (int *)(scratch + 64);
    double *d_pxy = (double *)(scratch + 256), *d_v = d_pxy + 4 * (size_t)g.A;
    VAH_TRY(cudaMemsetAsync(maxbits, 0, sizeof(unsigned long long), b->stream));
    VAH_TRY(vah::ic_participants_device(g.b, g.sigma_nn_fm2, g.A, g.ws_R, g.ws_a, g.seed, d_pxy, d_np, b->stream));
    VAH_TRY(vah::ic_deposit_device(d_pxy, d_np, g.width, lat.nx, lat.ny, lat.dx, lat.dy, d_v, maxbits, b->stream));
    int np = 0;  // the sampler reports -1 when its draws ran out (parameters it cannot sample)
    VAH_TRY(cudaMemcpyAsync(&np, d_np, sizeof(int), cudaMemcpyDeviceToHost, b->stream));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    if (np < 0) {
        VAH_TRY(cudaFreeAsync(scratch, b->stream));
        return VAH_ERR_ARG;
    }
    VAH_TRY(vah::ic_fill_device<S>(d_v, maxbits, lat.nx, lat.ny, lat.nz, d.ncx, lat.dz, g.eta_flat, g.sigma_eta,
                                   g.e_peak, g.e_floor, d.ep[0][0], b->stream));
    VAH_TRY(cudaFreeAsync(scratch, b->stream));
    return VAH_OK;
}

// Initial state of a slot: e interior uploaded (or generated on the device),
// p = EoS(e), u = 1, pi = 0, conserved variables, ghost layers (the
// vah_event_init_from_e sequence).
template <typename S>
int init_slot(vah_batch *b, int slot, double t0, const double *e_interior, const vah_glauber *glauber, int pl_mode) {
    vah_batch::Slot &sl = b->slots[slot];
    SlotDesc<S> &d = *desc_host<S>(b, slot);
    const int nx = sl.lat.nx, ny = sl.lat.ny, nz = sl.lat.nz;
    std::vector<S> stage;
    if (glauber) {
        const int rc = glauber_slot<S>(b, d, sl.lat, *glauber);
        if (rc != VAH_OK) return rc;
    } else {
        stage.resize((size_t)nx * ny * nz);
        for (size_t k = 0; k < stage.size(); ++k) stage[k] = (S)e_interior[k];
        for (int k = 0; k < nz; ++k) {
            S *dst = d.ep[0][0] + 2 + (size_t)d.ncx * (2 + (size_t)d.ncy * (k + 2));
            VAH_TRY(cudaMemcpy2DAsync(dst, d.ncx * sizeof(S), stage.data() + (size_t)nx * ny * k, nx * sizeof(S),
                                      nx * sizeof(S), ny, cudaMemcpyHostToDevice, b->stream));
        }
    }
    S *qs[16];
    for (int n = 0; n < 16; ++n) qs[n] = n < b->nq || (n == 15 && b->nq == 16) ? d.q[n] : nullptr;
    VAH_TRY(vah::launch_init_primitives<S>(fs<S>(qs, 16), fs<S>(d.uA, 4), d.ep[0][0], d.ep[0][1], batch_eos(b), nx, ny,
                                           nz, d.ncx, b->stream));
    VAH_TRY(vah::launch_set_conserved<S>(fs<S>(qs, 16), fs<S>(d.uA, 4), fs<S>(d.uB, 4), d.ep[0][0], b->opt.physics,
                                         nx, ny, nz, d.ncx, t0, pl_mode == VAH_PL_ISOTROPIC, b->stream));
    vah::FieldSet<S> g{};
    int m = 0;
    g.f[m++] = d.ep[0][0];
    g.f[m++] = d.ep[0][1];
    for (int k = 0; k < 4; ++k) g.f[m++] = d.uA[k];
    for (int k = 0; k < b->nq; ++k) g.f[m++] = d.q[k];
    g.n = m;
    VAH_TRY(vah::launch_ghosts<S>(g, nx, ny, nz, d.ncx, b->stream));
    SlotClock c{t0, 0, 1, 0};
    VAH_TRY(cudaMemcpyAsync(b->d_clk + slot, &c, sizeof(c), cudaMemcpyHostToDevice, b->stream));
    VAH_TRY(cudaMemcpyAsync(b->d_dt + slot, &sl.dt, sizeof(double), cudaMemcpyHostToDevice, b->stream));
    VAH_TRY(cudaMemsetAsync(b->d_counters + 4 * slot, 0, 4 * sizeof(unsigned long long), b->stream));
    VAH_TRY(cudaMemsetAsync(b->d_cross + 2 * slot, 0, 2 * sizeof(unsigned long long), b->stream));
    VAH_TRY(cudaMemsetAsync(b->d_vol + slot, 0, sizeof(double), b->stream));
    const double dv = sl.lat.dx * sl.lat.dy * sl.lat.dz;
    VAH_TRY(cudaMemcpyAsync(b->d_dv + slot, &dv, sizeof(double), cudaMemcpyHostToDevice, b->stream));
    vah::hot_init_kernel<S><<<std::max(1, std::min(nx * ny * nz / 256 + 1, 148 * 16)), 256, 0, b->stream>>>(
        d.ep[0][0], d.hot, d.e_freeze, nx, ny, nz, d.ncx);
    VAH_TRY(cudaGetLastError());
    VAH_TRY(cudaStreamSynchronize(b->stream));  // the staging vector dies here
    return VAH_OK;
}

// Device array currently holding a field of a slot.
template <typename S>
S *slot_field(vah_batch *b, int slot, int field, int parity) {
    SlotDesc<S> &d = *desc_host<S>(b, slot);
    if (field >= 0 && field < 16) return field < b->nq || (field == 15 && b->nq == 16) ? d.q[field] : nullptr;
    if (field == VAH_F_E) return d.ep[0][0];
    if (field == VAH_F_P) return d.ep[0][1];
    if (field >= VAH_F_UT && field <= VAH_F_UN) return (parity ? d.uB : d.uA)[field - VAH_F_UT];
    if (field >= VAH_F_UPT && field <= VAH_F_UPN) return (parity ? d.uA : d.uB)[field - VAH_F_UPT];
    return nullptr;
}

}  // namespace

extern "C" int vah_batch_create(const vah_options *opt, const double *eos_table, size_t capacity_bytes,
                                vah_batch **out) {
    if (!opt || !out) return VAH_ERR_ARG;
    *out = nullptr;
    if (opt->physics < VAH_IDEAL || opt->physics > VAH_PIMUNU_PI) return VAH_ERR_ARG;
    if (opt->eos == VAH_EOS_TABLE && !eos_table) return VAH_ERR_ARG;
    if (opt->precision != VAH_FP64 && opt->precision != VAH_FP32) return VAH_ERR_ARG;
    if (opt->flux != VAH_FLUX_PER_CELL && opt->flux != VAH_FLUX_SHARED) return VAH_ERR_ARG;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) return VAH_ERR_NODEVICE;
    if (opt->device < 0 || opt->device >= ndev) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(opt->device));
    vah_batch *b = new vah_batch();
    b->opt = *opt;
    b->nq = nq_of(opt->physics);
    b->elem = opt->precision == VAH_FP32 ? sizeof(float) : sizeof(double);
    b->own_stream = opt->stream == nullptr;
    b->capacity = capacity_bytes;
    b->used = 0;
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, opt->device);
    int rc = VAH_OK;
    auto chk = [&](cudaError_t e) {
        if (rc == VAH_OK && e != cudaSuccess) rc = cuda_status(e);
    };
    if (b->own_stream) chk(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
    else b->stream = (cudaStream_t)opt->stream;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = opt->device;
    chk(cudaMemPoolCreate(&b->pool, &props));
    if (rc == VAH_OK) {
        uint64_t keep = UINT64_MAX;  // keep freed event memory in the pool for the next admission
        cudaMemPoolSetAttribute(b->pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    const size_t desc_size = b->elem == sizeof(float) ? sizeof(SlotDesc<float>) : sizeof(SlotDesc<double>);
    b->desc_host.assign(desc_size * vah::kMaxSlots, 0);
    b->slots.resize(vah::kMaxSlots);
    chk(cudaMalloc(&b->d_desc, desc_size * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_clk, sizeof(SlotClock) * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_dt, sizeof(double) * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_cross, sizeof(unsigned long long) * 2 * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_vol, sizeof(double) * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_dv, sizeof(double) * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_counters, sizeof(unsigned long long) * 4 * vah::kMaxSlots));
    chk(cudaMalloc((void **)&b->d_maxbits, sizeof(unsigned long long) * vah::kMaxSlots));
    b->fstage = vah::kFieldStageValues;
    chk(cudaMalloc((void **)&b->d_fstage, sizeof(double) * b->fstage));
    if (rc == VAH_OK) {
        chk(cudaMemset(b->d_clk, 0, sizeof(SlotClock) * vah::kMaxSlots));
        chk(cudaMemset(b->d_dt, 0, sizeof(double) * vah::kMaxSlots));
        chk(cudaMemset(b->d_counters, 0, sizeof(unsigned long long) * 4 * vah::kMaxSlots));
        chk(cudaMemset(b->d_cross, 0, sizeof(unsigned long long) * 2 * vah::kMaxSlots));
        chk(cudaMemset(b->d_vol, 0, sizeof(double) * vah::kMaxSlots));
        chk(cudaMemset(b->d_dv, 0, sizeof(double) * vah::kMaxSlots));
    }
    if (rc == VAH_OK && opt->eos == VAH_EOS_TABLE) {
        const size_t len = VAH_EOS_TABLE_LEN((size_t)eos_table[0]);
        chk(cudaMalloc((void **)&b->d_tab, len * sizeof(double)));
        chk(cudaMemcpy(b->d_tab, eos_table, len * sizeof(double), cudaMemcpyHostToDevice));
        b->tab.assign(eos_table, eos_table + len);
    }
    if (rc == VAH_OK && opt->eos == VAH_EOS_CONFORMAL) {
        const std::vector<uint32_t> &exc = vah::powf_quarter_exceptions();
        b->nexc = (int)(exc.size() / 2);
        if (b->nexc) {
            chk(cudaMalloc((void **)&b->d_exc, exc.size() * sizeof(uint32_t)));
            chk(cudaMemcpy(b->d_exc, exc.data(), exc.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
        }
    }
    chk(cudaEventCreate(&b->t0));
    chk(cudaEventCreate(&b->t1));
    b->dirty = true;
    if (rc != VAH_OK) {
        delete b;  // device resources of a failed create are reclaimed at context teardown
        return rc;
    }
    *out = b;
    return VAH_OK;
}

extern "C" int vah_batch_destroy(vah_batch *b) {
    if (!b) return VAH_ERR_ARG;
    cudaSetDevice(b->opt.device);
    cudaStreamSynchronize(b->stream);
    if (b->has_graph) cudaGraphExecDestroy(b->graph);
    for (auto &sl : b->slots)
        if (sl.mem) cudaFreeAsync(sl.mem, b->stream);
    for (int k = 0; k < vah::K_NUM; ++k)
        if (b->d_work[k]) cudaFreeAsync(b->d_work[k], b->stream);
    if (b->d_partial) cudaFreeAsync(b->d_partial, b->stream);
    if (b->d_args) cudaFreeAsync(b->d_args, b->stream);
    if (b->d_scratch) cudaFreeAsync(b->d_scratch, b->stream);
    if (b->d_slabs) cudaFreeAsync(b->d_slabs, b->stream);
    cudaStreamSynchronize(b->stream);
    cudaMemPoolDestroy(b->pool);
    cudaFree(b->d_desc);
    cudaFree(b->d_clk);
    cudaFree(b->d_dt);
    cudaFree(b->d_cross);
    cudaFree(b->d_vol);
    cudaFree(b->d_dv);
    cudaFree(b->d_counters);
    cudaFree(b->d_maxbits);
    cudaFree(b->d_fstage);
    cudaFree(b->d_tab);
    cudaFree(b->d_exc);
    cudaEventDestroy(b->t0);
    cudaEventDestroy(b->t1);
    if (b->own_stream) cudaStreamDestroy(b->stream);
    delete b;
    return VAH_OK;
}

extern "C" int vah_batch_event_bytes(const vah_batch *b, const vah_lattice *lat, size_t *bytes) {
    if (!b || !lat || !bytes || lat->nx < 1 || lat->ny < 1 || lat->nz < 1) return VAH_ERR_ARG;
    *bytes = event_bytes(b, lat);
    return VAH_OK;
}

namespace {

// Admission shared by vah_batch_add and vah_batch_add_glauber: footprint
// check, slot memory, descriptors, initial state.
int add_slot(vah_batch *b, const vah_lattice *lat, const vah_hydro *hydro, double dt, const double *e_interior,
             const vah_glauber *glauber, int pl_mode, int *slot_out) {
    if (!b || !lat || !hydro || (!e_interior && !glauber) || !slot_out || !(dt > 0) || !(hydro->t0 > 0))
        return VAH_ERR_ARG;
    if (lat->nx < 1 || lat->ny < 1 || lat->nz < 1 || !(hydro->eta_over_s > 0)) return VAH_ERR_ARG;
    const size_t bytes = event_bytes(b, lat);
    if (b->used + bytes > b->capacity) return VAH_ERR_FULL;
    int slot = -1;
    for (int s = 0; s < vah::kMaxSlots; ++s)
        if (!b->slots[s].used) {
            slot = s;
            break;
        }
    if (slot < 0) return VAH_ERR_FULL;
    VAH_TRY(cudaSetDevice(b->opt.device));
    if ((size_t)lat->nx + 4 > b->fstage) {  // the staging holds a row of any event
        double *wider = nullptr;
        VAH_TRY(cudaStreamSynchronize(b->stream));
        VAH_TRY(cudaMalloc((void **)&wider, sizeof(double) * ((size_t)lat->nx + 4)));
        cudaFree(b->d_fstage);
        b->d_fstage = wider;
        b->fstage = (size_t)lat->nx + 4;
    }
    // the scratch: never less than the event needs, nor more than the room that it leaves
    const ScratchBounds sb = scratch_bounds(b, lat, b->capacity - b->used - bytes);
    int rc = VAH_OK;
    if (b->cap_scratch < sb.least || b->cap_scratch > sb.most)
        rc = set_scratch(b, std::min(std::max(sb.least, kScratchBeyond), sb.all), sb.least);
    if (rc != VAH_OK) return rc;
    vah_batch::Slot &sl = b->slots[slot];
    cudaError_t e = cudaMallocFromPoolAsync(&sl.mem, bytes, b->pool, b->stream);
    if (e == cudaErrorMemoryAllocation && b->cap_scratch > sb.least) {  // the scratch makes way
        cudaGetLastError();
        if ((rc = set_scratch(b, sb.least, sb.least)) != VAH_OK) return rc;
        e = cudaMallocFromPoolAsync(&sl.mem, bytes, b->pool, b->stream);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();  // else the next launch's check would find it
        sl.mem = nullptr;
        return cuda_status(e);
    }
    VAH_TRY(cudaMemsetAsync(sl.mem, 0, bytes, b->stream));
    sl.used = true;
    sl.lat = *lat;
    sl.hydro = *hydro;
    sl.dt = dt;
    sl.bytes = bytes;
    sl.admitted = b->steps;
    b->used += bytes;
    rc = b->elem == sizeof(float) ? fill_slot<float>(b, slot) : fill_slot<double>(b, slot);
    if (rc == VAH_OK)
        rc = b->elem == sizeof(float) ? init_slot<float>(b, slot, hydro->t0, e_interior, glauber, pl_mode)
                                      : init_slot<double>(b, slot, hydro->t0, e_interior, glauber, pl_mode);
    if (rc != VAH_OK) {
        vah_batch_remove(b, slot);
        return rc;
    }
    b->dirty = true;
    *slot_out = slot;
    return VAH_OK;
}

}  // namespace

extern "C" int vah_batch_add(vah_batch *b, const vah_lattice *lat, const vah_hydro *hydro, double dt,
                             const double *e_interior, int pl_mode, int *slot_out) {
    if (!e_interior) return VAH_ERR_ARG;
    return add_slot(b, lat, hydro, dt, e_interior, nullptr, pl_mode, slot_out);
}

extern "C" int vah_batch_add_glauber(vah_batch *b, const vah_lattice *lat, const vah_hydro *hydro, double dt,
                                     const vah_glauber *g, int pl_mode, int *slot_out) {
    if (!g || g->A < 1 || !(g->width > 0) || !(g->e_peak > 0) || !(g->e_floor >= 0)) return VAH_ERR_ARG;
    if (lat && lat->nz > 1 && !(g->sigma_eta > 0)) return VAH_ERR_ARG;
    return add_slot(b, lat, hydro, dt, nullptr, g, pl_mode, slot_out);
}

extern "C" int vah_batch_remove(vah_batch *b, int slot) {
    if (!b || slot < 0 || slot >= vah::kMaxSlots || !b->slots[slot].used) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    vah_batch::Slot &sl = b->slots[slot];
    SlotClock c{0.0, 0, 0, 0};
    VAH_TRY(cudaMemcpyAsync(b->d_clk + slot, &c, sizeof(c), cudaMemcpyHostToDevice, b->stream));
    VAH_TRY(cudaFreeAsync(sl.mem, b->stream));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    b->used -= sl.bytes;
    sl = vah_batch::Slot();
    b->dirty = true;
    return VAH_OK;
}

extern "C" int vah_batch_step(vah_batch *b, int nsteps) {
    if (!b || nsteps < 0) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    int rc;
    if (b->dirty) {
        if ((rc = rebuild(b)) != VAH_OK) return rc;
        if ((rc = capture_graph(b)) != VAH_OK) return rc;
    }
    if (b->timing) VAH_TRY(cudaEventRecord(b->t0, b->stream));
    for (int n = 0; n < nsteps; ++n) {
        VAH_TRY(cudaGraphLaunch(b->graph, b->stream));
        ++b->steps;
    }
    if (b->timing) {
        VAH_TRY(cudaEventRecord(b->t1, b->stream));
        VAH_TRY(cudaEventSynchronize(b->t1));
        float ms = 0;
        VAH_TRY(cudaEventElapsedTime(&ms, b->t0, b->t1));
        b->kernel_ms += ms;
        b->kernel_steps += nsteps;
    }
    return VAH_OK;
}

extern "C" int vah_batch_sync(vah_batch *b) {
    if (!b) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    return VAH_OK;
}

extern "C" int vah_batch_event_info(vah_batch *b, int slot, vah_event_info *out) {
    if (!b || !out || slot < 0 || slot >= vah::kMaxSlots || !b->slots[slot].used) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    SlotClock c;
    unsigned long long cnt[4];
    VAH_TRY(cudaMemcpyAsync(&c, b->d_clk + slot, sizeof(c), cudaMemcpyDeviceToHost, b->stream));
    VAH_TRY(cudaMemcpyAsync(cnt, b->d_counters + 4 * slot, sizeof(cnt), cudaMemcpyDeviceToHost, b->stream));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    out->t = c.t;
    out->steps = c.steps;
    out->face_fallbacks = (long long)cnt[0];
    out->cell_fallbacks = (long long)cnt[1];
    out->nan_cells = (long long)cnt[2];
    out->bytes = (long long)b->slots[slot].bytes;
    return VAH_OK;
}

template <typename S>
const unsigned char *slot_fallback(vah_batch *b, int slot) {
    return desc_host<S>(b, slot)->fallback;
}

extern "C" int vah_batch_get_field(vah_batch *b, int slot, int field, double *host, int with_ghosts) {
    if (!b || !host || slot < 0 || slot >= vah::kMaxSlots || !b->slots[slot].used) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    const vah_lattice &lat = b->slots[slot].lat;
    const int ncx = lat.nx + 4, parity = (int)((b->steps - b->slots[slot].admitted) & 1);
    auto read = [&](auto *src) -> int {
        using S = std::remove_reference_t<decltype(*src)>;
        if (!src) return VAH_ERR_ARG;
        if (with_ghosts && lat.nz == 1) {  // 2+1D steps leave the eta ghost layers to the reader
            vah::FieldSet<S> f{};
            f.f[0] = src;
            f.n = 1;
            VAH_TRY(vah::launch_ghost_pass<S>(f, lat.nx, lat.ny, lat.nz, ncx, 2, b->stream));
        }
        VAH_TRY(vah::read_field<S>(src, host, lat.nx, lat.ny, lat.nz, ncx, with_ghosts != 0, b->d_fstage, b->fstage,
                                   b->stream));
        VAH_TRY(cudaStreamSynchronize(b->stream));
        return VAH_OK;
    };
    return b->elem == sizeof(float) ? read(slot_field<float>(b, slot, field, parity))
                                    : read(slot_field<double>(b, slot, field, parity));
}

extern "C" int vah_batch_fallback_mask(vah_batch *b, int slot, unsigned char *host) {
    if (!b || !host || slot < 0 || slot >= vah::kMaxSlots || !b->slots[slot].used) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    const vah_lattice &lat = b->slots[slot].lat;
    const size_t ncx = lat.nx + 4, ncy = lat.ny + 4;
    const unsigned char *src = b->elem == sizeof(float) ? slot_fallback<float>(b, slot) : slot_fallback<double>(b, slot);
    for (int k = 0; k < lat.nz; ++k)
        VAH_TRY(cudaMemcpy2DAsync(host + (size_t)lat.nx * lat.ny * k, lat.nx, src + 2 + ncx * (2 + ncy * (k + 2)), ncx,
                                  lat.nx, lat.ny, cudaMemcpyDeviceToHost, b->stream));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    return VAH_OK;
}

extern "C" int vah_batch_freezeout_volume(vah_batch *b, double *out, int nslots) {
    if (!b || !out || nslots < 0 || nslots > vah::kMaxSlots) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    if (nslots) VAH_TRY(cudaMemcpy(out, b->d_vol, sizeof(double) * nslots, cudaMemcpyDeviceToHost));
    for (int s = 0; s < nslots; ++s)
        if (s >= (int)b->slots.size() || !b->slots[s].used) out[s] = 0.0;
    return VAH_OK;
}

extern "C" int vah_batch_max_energy_density(vah_batch *b, double *out, int nslots) {
    if (!b || !out || nslots < 1) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    int rc;
    if (b->dirty && (rc = rebuild(b)) != VAH_OK) return rc;
    VAH_TRY(cudaMemsetAsync(b->d_maxbits, 0, sizeof(unsigned long long) * vah::kMaxSlots, b->stream));
    for (int kind : {vah::K_C2, vah::K_C3}) {
        if (!b->nwork[kind]) continue;
        const int grid = std::min(b->nwork[kind], b->sms * 8);
        if (b->elem == sizeof(float))
            vah::max_e_kernel<float><<<grid, dim3(vah::kTX, vah::kTY), 0, b->stream>>>(
                (const SlotDesc<float> *)b->d_desc, b->d_work[kind], b->nwork[kind], b->d_maxbits, 0);
        else
            vah::max_e_kernel<double><<<grid, dim3(vah::kTX, vah::kTY), 0, b->stream>>>(
                (const SlotDesc<double> *)b->d_desc, b->d_work[kind], b->nwork[kind], b->d_maxbits, 0);
        VAH_TRY(cudaGetLastError());
    }
    std::vector<unsigned long long> bits(vah::kMaxSlots);
    VAH_TRY(cudaMemcpyAsync(bits.data(), b->d_maxbits, bits.size() * sizeof(unsigned long long),
                            cudaMemcpyDeviceToHost, b->stream));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    for (int s = 0; s < nslots && s < vah::kMaxSlots; ++s) {
        double v;
        memcpy(&v, &bits[s], sizeof(v));
        out[s] = b->slots[s].used ? v : 0.0;
    }
    return VAH_OK;
}

extern "C" int vah_batch_observables(vah_batch *b, double *out, int nslots) {
    if (!b || !out || nslots < 1) return VAH_ERR_ARG;
    VAH_TRY(cudaSetDevice(b->opt.device));
    int rc;
    if (b->dirty && (rc = rebuild(b)) != VAH_OK) return rc;
    const int n2 = b->nwork[vah::K_C2], n3 = b->nwork[vah::K_C3];
    auto launch = [&](int kind, double *part) -> cudaError_t {
        const int nw = b->nwork[kind];
        if (!nw) return cudaSuccess;
        const int grid = std::min(nw, b->sms * 8);
        const dim3 blk(vah::kTX, vah::kTY);
        const bool f = b->elem == sizeof(float);
        switch (b->opt.physics) {
        case VAH_IDEAL:
            if (f) vah::observables_kernel<float, 0><<<grid, blk, 0, b->stream>>>((const SlotDesc<float> *)b->d_desc, b->d_clk, b->d_work[kind], nw, part);
            else vah::observables_kernel<double, 0><<<grid, blk, 0, b->stream>>>((const SlotDesc<double> *)b->d_desc, b->d_clk, b->d_work[kind], nw, part);
            break;
        case VAH_PIMUNU:
            if (f) vah::observables_kernel<float, 1><<<grid, blk, 0, b->stream>>>((const SlotDesc<float> *)b->d_desc, b->d_clk, b->d_work[kind], nw, part);
            else vah::observables_kernel<double, 1><<<grid, blk, 0, b->stream>>>((const SlotDesc<double> *)b->d_desc, b->d_clk, b->d_work[kind], nw, part);
            break;
        default:
            if (f) vah::observables_kernel<float, 2><<<grid, blk, 0, b->stream>>>((const SlotDesc<float> *)b->d_desc, b->d_clk, b->d_work[kind], nw, part);
            else vah::observables_kernel<double, 2><<<grid, blk, 0, b->stream>>>((const SlotDesc<double> *)b->d_desc, b->d_clk, b->d_work[kind], nw, part);
        }
        return cudaGetLastError();
    };
    VAH_TRY(launch(vah::K_C2, b->d_partial));
    VAH_TRY(launch(vah::K_C3, b->d_partial + (size_t)n2 * 5));
    std::vector<double> part((size_t)(n2 + n3) * 5);
    std::vector<WorkItem> w2(n2), w3(n3);
    if (n2 + n3) VAH_TRY(cudaMemcpyAsync(part.data(), b->d_partial, part.size() * sizeof(double), cudaMemcpyDeviceToHost, b->stream));
    if (n2) VAH_TRY(cudaMemcpyAsync(w2.data(), b->d_work[vah::K_C2], n2 * sizeof(WorkItem), cudaMemcpyDeviceToHost, b->stream));
    if (n3) VAH_TRY(cudaMemcpyAsync(w3.data(), b->d_work[vah::K_C3], n3 * sizeof(WorkItem), cudaMemcpyDeviceToHost, b->stream));
    VAH_TRY(cudaStreamSynchronize(b->stream));
    std::vector<double> acc((size_t)nslots * 5, 0.0);
    auto add = [&](const std::vector<WorkItem> &w, size_t base) {
        for (size_t k = 0; k < w.size(); ++k)
            if (w[k].slot < nslots)
                for (int m = 0; m < 5; ++m) acc[(size_t)w[k].slot * 5 + m] += part[(base + k) * 5 + m];
    };
    add(w2, 0);
    add(w3, n2);
    for (int s = 0; s < nslots; ++s) {
        const double *a = &acc[(size_t)s * 5];
        out[3 * s + 0] = a[0];
        out[3 * s + 1] = a[2] != 0 ? a[1] / a[2] : 0.0;
        out[3 * s + 2] = a[4] != 0 ? a[3] / a[4] : 0.0;
    }
    return VAH_OK;
}

extern "C" int vah_batch_set_timing(vah_batch *b, int on) {
    if (!b) return VAH_ERR_ARG;
    b->timing = on != 0;
    return VAH_OK;
}

extern "C" int vah_batch_kernel_time(vah_batch *b, double *ms, long long *steps) {
    if (!b || !ms || !steps) return VAH_ERR_ARG;
    *ms = b->kernel_ms;
    *steps = b->kernel_steps;
    b->kernel_ms = 0;
    b->kernel_steps = 0;
    return VAH_OK;
}

namespace {

// The batch form of vah_event_autotune: times the flux launch (reported as the
// first of the three flux kinds) and the cell launches of the first group,
// `reps` times in stage-1 buffer roles (outputs are stage scratch); each has
// one configuration. The per-slot counters are restored.
int batch_autotune(vah_batch *b, int reps, vah_tune_report *out) {
    using namespace vah;
    std::vector<unsigned long long> saved((size_t)kMaxSlots * 4);
    VAH_TRY(cudaStreamSynchronize(b->stream));
    VAH_TRY(cudaMemcpy(saved.data(), b->d_counters, saved.size() * sizeof(unsigned long long),
                       cudaMemcpyDeviceToHost));
    int rc = launch_args(b);
    if (rc != VAH_OK) return rc;
    cudaEvent_t e0, e1;
    VAH_TRY(cudaEventCreate(&e0));
    VAH_TRY(cudaEventCreate(&e1));
    out->nkinds = 5;
    for (int kind = 0; kind < 5 && rc == VAH_OK; ++kind) {
        const int list = kind < 3 ? K_FLUX : (kind == 3 ? K_C2 : K_C3);
        out->kind[kind] = {kTX, kTY, kind == 3 ? 3 : 4, 0.0, 0.0};
        if (kind == 1 || kind == 2 || b->groups.empty() || b->groups[0].count[list] == 0) continue;
        auto launch = [&]() { return launch_list_any(b, b->groups[0], list, 1) == cudaSuccess; };
        bool ok = launch() && cudaEventRecord(e0, b->stream) == cudaSuccess;
        for (int k = 0; k < reps && ok; ++k) ok = launch();
        float f = 0;
        if (!ok || cudaEventRecord(e1, b->stream) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
            cudaEventElapsedTime(&f, e0, e1) != cudaSuccess)
            rc = VAH_ERR_CUDA;
        out->kind[kind].ms_default = out->kind[kind].ms_best = f / reps;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (cudaMemcpy(b->d_counters, saved.data(), saved.size() * sizeof(unsigned long long),
                   cudaMemcpyHostToDevice) != cudaSuccess &&
        rc == VAH_OK)
        rc = VAH_ERR_CUDA;
    return rc;
}

}  // namespace

extern "C" int vah_batch_autotune(vah_batch *b, int reps, vah_tune_report *out) {
    if (!b || !out || reps < 1) return VAH_ERR_ARG;
    memset(out, 0, sizeof(*out));
    if (b->elem == sizeof(float)) return VAH_OK;  // the FP32 form has nothing to tune
    VAH_TRY(cudaSetDevice(b->opt.device));
    if (b->dirty) {  // the work-list must describe the admitted events
        const int rc = rebuild(b);
        if (rc != VAH_OK) return rc;
    }
    return batch_autotune(b, reps, out);
}
