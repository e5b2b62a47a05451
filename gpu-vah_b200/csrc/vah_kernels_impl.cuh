// vah_kernels_impl.cuh -- CUDA kernels of the VAH time step (sm_100a) and
// their launch dispatch. Compiled once per storage type by vah_kernels_f64.cu
// and vah_kernels_f32.cu (separate translation units build in parallel).
//
// stage_kernel: one thread per interior cell runs the whole RK stage of that
// cell (vah_stage.cuh; FP64). flux_kernel + cell_kernel: the same stage split
// into one launch for the flux differences along every axis (vah_march.cuh)
// and one for the cells (the default path, and the FP32 form). 128-
// or 64-thread blocks, x fastest so that the loads of a field coalesce.
#pragma once

#include "vah_kernels.cuh"
#include "vah_march.cuh"
#include "vah_tile_cell.cuh"

namespace vah {

namespace {

constexpr int kBX = 32, kBY = 4;  // fused stage kernel shape

// Row blocks beyond the grid's y limit (65535) continue along z.
constexpr unsigned kMaxGridY = 65535;

__device__ __forceinline__ int row_block() { return (int)(blockIdx.z * gridDim.y + blockIdx.y); }

dim3 row_grid(long long cols, long long rows, int bx, int by) {
    const unsigned gy = (unsigned)((rows + by - 1) / by);
    const unsigned gz = (gy + kMaxGridY - 1) / kMaxGridY;
    return dim3((unsigned)((cols + bx - 1) / bx), gz > 1 ? kMaxGridY : gy, gz > 1 ? gz : 1);
}

template <typename S, int PHYS, bool IS3D>
__global__ void __launch_bounds__(kBX *kBY) stage_kernel(const StageArgs<S> a) {
    const int i = blockIdx.x * kBX + threadIdx.x;
    const int r = row_block() * kBY + threadIdx.y;  // row index over (j, k)
    if (i >= a.nx || r >= a.ny * a.nz) return;
    const int j = r % a.ny, k = r / a.ny;
    stage_cell<S, PHYS, IS3D>(a, i + 2, j + 2, k + 2);
}

// What the blocks of one flux launch do: eta marches first, then y marches (the
// long ones), then x strips, which fill the tail.
struct FluxGrid {
    int zblocks, yblocks, xblocks;
    int zstrips, zseg, ystrips, yseg, xstrips;
};

// The flux differences of the planes [k0, k1): a warp per x strip, or per
// strip and segment of a march.
template <typename S, int PHYS, bool EXACT>
__global__ void __launch_bounds__(kFluxThreads, kFluxMinb<S>) flux_kernel(const StageArgs<S> a, const FluxGrid g) {
    extern __shared__ __align__(16) unsigned char flux_sm[];
    after_previous_launch();
    const SelectPointers<S, PHYS> sel{a};
    const int warp = threadIdx.x / 32;
    int block = blockIdx.x;
    S *sm = (S *)flux_sm + warp * kMarchValues<S, PHYS>;
    if (block < g.zblocks) {
        const int w = block * 4 + warp, part = w / g.zstrips, m0 = a.k0 + part * g.zseg;
        if (m0 < a.k1)
            flux_march<PHYS, 2, EXACT>(a, sel, w - part * g.zstrips, m0, min(m0 + g.zseg, a.k1), sm);
        return;
    }
    block -= g.zblocks;
    if (block < g.yblocks) {
        const int w = block * 4 + warp, part = w / g.ystrips, m0 = part * g.yseg;
        if (m0 < a.ny)
            flux_march<PHYS, 1, EXACT>(a, sel, w - part * g.ystrips, m0, min(m0 + g.yseg, a.ny), sm);
        return;
    }
    block -= g.yblocks;
    if constexpr (Lanes<S, PHYS>::SPLIT) {
        __shared__ TablePointers<S> tab;
        set_table_pointers<PHYS>(tab, a, threadIdx.x);
        __syncthreads();
        if (block * 4 + warp < g.xstrips) flux_x<PHYS, EXACT>(a, tab, block * 4 + warp);
    } else if (block * 4 + warp < g.xstrips) {
        flux_x<PHYS, EXACT>(a, sel, block * 4 + warp);
    }
}

// One warp per row at a time; PACK: device layout -> packed, else back.
template <typename S, bool PACK>
__global__ void pack_kernel(S *__restrict__ field, double *__restrict__ packed, int w, int nyr, int pitch, int ncy,
                            int off, long long row0, long long rows) {
    for (long long r = blockIdx.x * (long long)blockDim.y + threadIdx.y; r < rows; r += (long long)gridDim.x * blockDim.y) {
        const long long k = (row0 + r) / nyr;
        const int j = (int)((row0 + r) - k * nyr);
        S *f = field + off + pitch * ((j + off) + (long long)ncy * (k + off));
        double *p = packed + r * w;
        for (int i = threadIdx.x; i < w; i += 32) {
            if (PACK) p[i] = (double)f[i];
            else f[i] = (S)p[i];
        }
    }
}

// Cells of the planes [k0, k1) in order, x fastest: a row's end does not idle
// the lanes of a warp (rows of 81 left 15 of 96 idle as 32-wide tiles).
template <typename S, int PHYS, bool IS3D>
__global__ void __launch_bounds__(kCellThreads, kCellMinb<S, IS3D>) cell_kernel(const StageArgs<S> a) {
    const int c = blockIdx.x * kCellThreads + threadIdx.x;
    after_previous_launch();
    if (c >= a.nx * a.ny * (a.k1 - a.k0)) return;
    const int r = c / a.nx, i = c - r * a.nx, k = r / a.ny, j = r - k * a.ny;
    if constexpr (sizeof(S) == 4) cell_compute_f32<PHYS, IS3D>(a, i + 2, j + 2, k + a.k0 + 2);
    else cell_compute<S, PHYS, IS3D, true>(a, i + 2, j + 2, k + a.k0 + 2);
}

template <typename S, int PHYS>
__global__ void validity_kernel(const ValidityArgs<S> a) {
    const long long n = (long long)a.nx * a.ny * a.nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % a.nx), j = (int)((c / a.nx) % a.ny), k = (int)(c / ((long long)a.nx * a.ny));
        validity_cell<S, PHYS>(a, (i + 2) + (long long)a.ncx * (j + 2) + a.plane * (k + 2));
    }
}

template <typename S, int PHYS>
__global__ void set_conserved_kernel(const FieldSet<S> q, const FieldSet<S> u, const FieldSet<S> up, const S *e,
                                     int nx, int ny, int nz, int pitch, double t, int pl_from_field) {
    const long long n = (long long)nx * ny * nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % nx), j = (int)((c / nx) % ny), k = (int)(c / ((long long)nx * ny));
        const long long s = (i + 2) + (long long)pitch * ((j + 2) + (long long)(ny + 4) * (k + 2));
        set_conserved_cell<S, PHYS>(q.f, u.f, up.f, e, t, pl_from_field, s);
    }
}

template <typename S>
__global__ void init_primitives_kernel(const FieldSet<S> q, const FieldSet<S> u, const S *e, S *p, const Eos eos,
                                       int nx, int ny, int nz, int pitch) {
    const long long n = (long long)nx * ny * nz;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(c % nx), j = (int)((c / nx) % ny), k = (int)(c / ((long long)nx * ny));
        const long long s = (i + 2) + (long long)pitch * ((j + 2) + (long long)(ny + 4) * (k + 2));
        const double pv = eos_pressure(eos, (double)e[s]);
        p[s] = (S)pv;
        u.f[0][s] = (S)1.0;
        u.f[1][s] = u.f[2][s] = u.f[3][s] = (S)0.0;
        for (int m = 5; m < 16; ++m)
            if (q.f[m]) q.f[m][s] = (S)0.0;
        q.f[kSlotPL][s] = (S)pv;
    }
}

// Pass 0 (I): j in [2, ncy), k in [2, ncz): i = 0,1 <- 2; i = nx+2, nx+3 <- nx+1.
// Pass 1 (J): i in [2, ncx), k in [2, ncz).  Pass 2 (K): i in [2, ncx), j in [2, ncy).
template <typename S>
__global__ void ghost_kernel(const FieldSet<S> f, int nx, int ny, int nz, int pitch, int pass) {
    const int ncx = nx + 4, ncy = ny + 4, ncz = nz + 4;
    const long long plane = (long long)pitch * ncy;
    int na, nb;
    if (pass == 0) { na = ncy - 2; nb = ncz - 2; }
    else if (pass == 1) { na = ncx - 2; nb = ncz - 2; }
    else { na = ncx - 2; nb = ncy - 2; }
    const long long n = (long long)na * nb * 4;
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const int slot = (int)(c & 3);
        const long long ab = c >> 2;
        const int A = (int)(ab % na) + 2, B = (int)(ab / na) + 2;
        long long s, sb;
        if (pass == 0) {
            int gi = slot < 2 ? slot : nx + slot, bi = slot < 2 ? 2 : nx + 1;
            s = gi + (long long)pitch * A + plane * B;
            sb = bi + (long long)pitch * A + plane * B;
        } else if (pass == 1) {
            int gj = slot < 2 ? slot : ny + slot, bj = slot < 2 ? 2 : ny + 1;
            s = A + (long long)pitch * gj + plane * B;
            sb = A + (long long)pitch * bj + plane * B;
        } else {
            int gk = slot < 2 ? slot : nz + slot, bk = slot < 2 ? 2 : nz + 1;
            s = A + (long long)pitch * B + plane * gk;
            sb = A + (long long)pitch * B + plane * bk;
        }
        for (int m = 0; m < f.n; ++m) f.f[m][s] = f.f[m][sb];
    }
}

template <typename S, int PHYS>
cudaError_t stage_dispatch(const StageArgs<S> &a, cudaStream_t stream) {
    dim3 block(kBX, kBY);
    const dim3 grid = row_grid(a.nx, (long long)a.ny * a.nz, kBX, kBY);
    if (a.nz > 1)
        stage_kernel<S, PHYS, true><<<grid, block, 0, stream>>>(a);
    else
        stage_kernel<S, PHYS, false><<<grid, block, 0, stream>>>(a);
    return cudaGetLastError();
}

// The flux launch; kind kFaceX, kFaceY or kFaceZ: that axis alone (for timing it), kCell: all.
template <typename S, int PHYS, bool EXACT>
cudaError_t flux_launch(const StageArgs<S> &a, int kind, cudaStream_t stream) {
    constexpr size_t smem = kFluxThreads / 32 * kMarchValues<S, PHYS> * sizeof(S);
    auto kernel = flux_kernel<S, PHYS, EXACT>;
    static_assert(smem <= 48 * 1024, "within the default shared memory limit");
    const int planes = a.k1 - a.k0;
    FluxGrid g{};
    if (kind == kFaceX || kind == kCell) {
        g.xstrips = flux_x_strips<S>(a.nx, a.ny, planes);
        g.xblocks = (g.xstrips + 3) / 4;
    }
    auto march = [&](int columns, int n, int &strips, int &seg, int &blocks) {
        strips = march_strips<S>(columns);
        seg = march_segment(n, kFluxMinb<S>, [&](int len) { return (long long)strips * ((n + len - 1) / len); });
        blocks = (strips * ((n + seg - 1) / seg) + 3) / 4;
    };
    if (kind == kFaceY || kind == kCell) march(a.nx * planes, a.ny, g.ystrips, g.yseg, g.yblocks);
    if (a.nz > 1 && (kind == kFaceZ || kind == kCell)) march(a.nx * a.ny, planes, g.zstrips, g.zseg, g.zblocks);
    const int grid = g.xblocks + g.yblocks + g.zblocks;
    if (grid == 0) return cudaSuccess;
    return launch_stage_kernel(kernel, follows_closely(a), grid, kFluxThreads, smem, stream, a, g);
}

template <typename S, int PHYS, bool IS3D>
cudaError_t cell_launch(const StageArgs<S> &a, cudaStream_t stream) {
    const int cells = a.nx * a.ny * (a.k1 - a.k0);
    return launch_stage_kernel(cell_kernel<S, PHYS, IS3D>, follows_closely(a), (cells + kCellThreads - 1) / kCellThreads, kCellThreads, 0, stream, a);
}

template <typename S, int PHYS>
cudaError_t kind_dispatch(const StageArgs<S> &a, bool exact, int kind, cudaStream_t stream) {
    if (kind == kCell) return a.nz > 1 ? cell_launch<S, PHYS, true>(a, stream) : cell_launch<S, PHYS, false>(a, stream);
    if constexpr (sizeof(S) == 8)
        if (exact) return flux_launch<S, PHYS, true>(a, kind, stream);
    return flux_launch<S, PHYS, false>(a, kind, stream);
}

// The arguments of one slab [k0, k1) of planes that the difference buffers
// hold: plane k0 is D's first.
template <typename S>
StageArgs<S> slab_args(const StageArgs<S> &a0, int k0, int k1) {
    StageArgs<S> a = a0;
    a.k0 = k0;
    a.k1 = k1;
    if (a0.d_planes > 0)
        for (int d = 0; d < 3; ++d)
            for (int n = 0; n < 16; ++n)
                if (a.D[d][n]) a.D[d][n] -= a.plane * (k0 + 2);
    return a;
}

// The stage of the planes [k0, k1), a slab at a time: each slab reads stage
// inputs only and writes stage outputs, so their order is free.
template <typename S, int PHYS>
cudaError_t stage_split_dispatch(const StageArgs<S> &a0, bool exact, cudaStream_t stream) {
    if (a0.k0 < 0 || a0.k1 > a0.nz || a0.k0 > a0.k1) return cudaErrorInvalidValue;
    const int slab = a0.d_planes > 0 ? a0.d_planes : a0.nz;
    for (int k0 = a0.k0; k0 < a0.k1; k0 += slab) {
        const StageArgs<S> a = slab_args(a0, k0, k0 + slab < a0.k1 ? k0 + slab : a0.k1);
        cudaError_t e;
        if constexpr (sizeof(S) == 8)
            e = exact ? flux_launch<S, PHYS, true>(a, kCell, stream) : flux_launch<S, PHYS, false>(a, kCell, stream);
        else
            e = flux_launch<S, PHYS, false>(a, kCell, stream);
        if (e == cudaSuccess) e = kind_dispatch<S, PHYS>(a, exact, kCell, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

int grid_for(long long n, int block) {
    long long g = (n + block - 1) / block;
    if (g > 148 * 64) g = 148 * 64;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace

template <typename S>
cudaError_t launch_stage(const StageArgs<S> &a, int physics, cudaStream_t stream) {
    switch (physics) {
    case kIdeal: return stage_dispatch<S, kIdeal>(a, stream);
    case kPimunu: return stage_dispatch<S, kPimunu>(a, stream);
    case kPimunuPi: return stage_dispatch<S, kPimunuPi>(a, stream);
    default: return cudaErrorInvalidValue;
    }
}

template <typename S>
cudaError_t launch_split_kind(const StageArgs<S> &a0, int physics, bool exact, int kind, cudaStream_t stream) {
    const StageArgs<S> a = slab_args(a0, a0.k0, a0.d_planes > 0 && a0.k0 + a0.d_planes < a0.k1 ? a0.k0 + a0.d_planes : a0.k1);
    switch (physics) {
    case kIdeal: return kind_dispatch<S, kIdeal>(a, exact, kind, stream);
    case kPimunu: return kind_dispatch<S, kPimunu>(a, exact, kind, stream);
    case kPimunuPi: return kind_dispatch<S, kPimunuPi>(a, exact, kind, stream);
    default: return cudaErrorInvalidValue;
    }
}

template <typename S>
cudaError_t launch_stage_split(const StageArgs<S> &a, int physics, bool exact, cudaStream_t stream) {
    switch (physics) {
    case kIdeal: return stage_split_dispatch<S, kIdeal>(a, exact, stream);
    case kPimunu: return stage_split_dispatch<S, kPimunu>(a, exact, stream);
    case kPimunuPi: return stage_split_dispatch<S, kPimunuPi>(a, exact, stream);
    default: return cudaErrorInvalidValue;
    }
}

template <typename S>
cudaError_t launch_validity(const ValidityArgs<S> &a, int physics, cudaStream_t stream) {
    const int block = 128, grid = grid_for((long long)a.nx * a.ny * a.nz, block);
    switch (physics) {
    case kIdeal: validity_kernel<S, kIdeal><<<grid, block, 0, stream>>>(a); break;
    case kPimunu: validity_kernel<S, kPimunu><<<grid, block, 0, stream>>>(a); break;
    case kPimunuPi: validity_kernel<S, kPimunuPi><<<grid, block, 0, stream>>>(a); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_set_conserved(const FieldSet<S> &q, const FieldSet<S> &u, const FieldSet<S> &up, const S *e,
                                 int physics, int nx, int ny, int nz, int pitch, double t, int pl_from_field,
                                 cudaStream_t stream) {
    const int block = 256;
    const int grid = grid_for((long long)nx * ny * nz, block);
    switch (physics) {
    case kIdeal: set_conserved_kernel<S, kIdeal><<<grid, block, 0, stream>>>(q, u, up, e, nx, ny, nz, pitch, t, pl_from_field); break;
    case kPimunu: set_conserved_kernel<S, kPimunu><<<grid, block, 0, stream>>>(q, u, up, e, nx, ny, nz, pitch, t, pl_from_field); break;
    case kPimunuPi: set_conserved_kernel<S, kPimunuPi><<<grid, block, 0, stream>>>(q, u, up, e, nx, ny, nz, pitch, t, pl_from_field); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_init_primitives(const FieldSet<S> &q, const FieldSet<S> &u, const S *e, S *p, const Eos &eos,
                                   int nx, int ny, int nz, int pitch, cudaStream_t stream) {
    const int block = 256;
    init_primitives_kernel<S><<<grid_for((long long)nx * ny * nz, block), block, 0, stream>>>(q, u, e, p, eos, nx, ny,
                                                                                                nz, pitch);
    return cudaGetLastError();
}

template <typename S>
cudaError_t launch_ghosts(const FieldSet<S> &fields, int nx, int ny, int nz, int pitch, cudaStream_t stream) {
    const int block = 256;
    for (int pass = 0; pass < 3; ++pass) {
        long long n;
        if (pass == 0) n = (long long)ny * nz;
        else if (pass == 1) n = (long long)nx * nz;
        else n = (long long)nx * ny;
        n = (n + 4LL * (nx + ny + nz) + 16) * 4;  // the passes also sweep upper ghost rows
        ghost_kernel<S><<<grid_for(n, block), block, 0, stream>>>(fields, nx, ny, nz, pitch, pass);
        cudaError_t err = cudaGetLastError();
        if (err != cudaSuccess) return err;
    }
    return cudaSuccess;
}

template <typename S, bool PACK>
cudaError_t pack_dispatch(S *field, double *packed, int nx, int ny, int pitch, bool ghosts, long long row0,
                          long long rows, cudaStream_t stream) {
    if (rows <= 0) return cudaSuccess;
    const int off = ghosts ? 0 : 2, grid = grid_for(rows, 8);
    pack_kernel<S, PACK><<<grid, dim3(32, 8), 0, stream>>>(field, packed, ghosts ? nx + 4 : nx, ghosts ? ny + 4 : ny,
                                                           pitch, ny + 4, off, row0, rows);
    return cudaGetLastError();
}
template <typename S>
cudaError_t launch_pack(const S *field, double *packed, int nx, int ny, int pitch, bool ghosts, long long row0,
                        long long rows, cudaStream_t stream) {
    return pack_dispatch<S, true>(const_cast<S *>(field), packed, nx, ny, pitch, ghosts, row0, rows, stream);
}
template <typename S>
cudaError_t launch_unpack(S *field, const double *packed, int nx, int ny, int pitch, bool ghosts, long long row0,
                          long long rows, cudaStream_t stream) {
    return pack_dispatch<S, false>(field, const_cast<double *>(packed), nx, ny, pitch, ghosts, row0, rows, stream);
}

// One pass of the ghost fill (0: x, 1: y, 2: eta), as launch_ghosts runs it.
template <typename S>
cudaError_t launch_ghost_pass(const FieldSet<S> &fields, int nx, int ny, int nz, int pitch, int pass,
                              cudaStream_t stream) {
    const int block = 256;
    long long n = pass == 0 ? (long long)ny * nz : (pass == 1 ? (long long)nx * nz : (long long)nx * ny);
    n = (n + 4LL * (nx + ny + nz) + 16) * 4;
    ghost_kernel<S><<<grid_for(n, block), block, 0, stream>>>(fields, nx, ny, nz, pitch, pass);
    return cudaGetLastError();
}

#define VAH_INSTANTIATE_SETUP(S)                                                                                \
    template cudaError_t launch_validity<S>(const ValidityArgs<S> &, int, cudaStream_t);                        \
    template cudaError_t launch_set_conserved<S>(const FieldSet<S> &, const FieldSet<S> &, const FieldSet<S> &, \
                                                 const S *, int, int, int, int, int, double, int, cudaStream_t); \
    template cudaError_t launch_init_primitives<S>(const FieldSet<S> &, const FieldSet<S> &, const S *, S *,    \
                                                   const Eos &, int, int, int, int, cudaStream_t);             \
    template cudaError_t launch_pack<S>(const S *, double *, int, int, int, bool, long long, long long,         \
                                        cudaStream_t);                                                          \
    template cudaError_t launch_unpack<S>(S *, const double *, int, int, int, bool, long long, long long,       \
                                          cudaStream_t);                                                        \
    template cudaError_t launch_ghosts<S>(const FieldSet<S> &, int, int, int, int, cudaStream_t);              \
    template cudaError_t launch_ghost_pass<S>(const FieldSet<S> &, int, int, int, int, int, cudaStream_t);
#define VAH_INSTANTIATE_SPLIT(S)                                                                                \
    template cudaError_t launch_split_kind<S>(const StageArgs<S> &, int, bool, int, cudaStream_t);              \
    template cudaError_t launch_stage_split<S>(const StageArgs<S> &, int, bool, cudaStream_t);

}  // namespace vah
