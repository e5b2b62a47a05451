// vah_kernels_impl.cuh -- CUDA kernels of the VAH time step (sm_100a) and
// their launch dispatch. Compiled once per storage type by vah_kernels_f64.cu
// and vah_kernels_f32.cu (separate translation units build in parallel).
//
// stage_kernel: one thread per interior cell runs the whole RK stage of that
// cell (vah_stage.cuh). flux_x_kernel + flux_march_kernel + cell_kernel: the
// same stage split into per-axis flux launches (vah_march.cuh) and one cell
// launch (the default path). 128-thread blocks, x fastest so that every load
// of a field is a coalesced row. The cell kernel takes its block shape at run
// time; the autotuner picks it by timing on the event's own state.
#pragma once

#include "vah_kernels.cuh"
#include "vah_march.cuh"

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

// The x flux differences of the planes [k0, k1): a warp per strip.
template <int PHYS, bool EXACT>
__global__ void __launch_bounds__(kSplitThreads, kFluxXMinb) flux_x_kernel(const StageArgs<double> a, int strips) {
    __shared__ HalfPointers hp;
    set_half_pointers<PHYS>(hp, a, threadIdx.x);
    __syncthreads();
    const int strip = blockIdx.x * (kSplitThreads / 32) + threadIdx.x / 32;
    if (strip < strips) flux_x<PHYS, EXACT>(a, hp, strip);
}

// The y or eta flux differences: a warp per strip and segment of `seg` cells.
template <int PHYS, int DIR, bool EXACT>
__global__ void __launch_bounds__(kSplitThreads, kMarchMinb) flux_march_kernel(const StageArgs<double> a, int strips, int seg) {
    extern __shared__ double march_sm[];
    const int lo = DIR == 1 ? 0 : a.k0, hi = DIR == 1 ? a.ny : a.k1;
    const int w = blockIdx.x * (kSplitThreads / 32) + threadIdx.x / 32;
    const int part = w / strips, m0 = lo + part * seg;
    if (m0 >= hi) return;
    flux_march<PHYS, DIR, EXACT>(a, HalfSelect<PHYS>{a}, w - part * strips, m0, min(m0 + seg, hi), march_sm + (threadIdx.x / 32) * kMarchDoubles<PHYS>);
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

template <int PHYS, bool IS3D>
__global__ void __launch_bounds__(kSplitThreads, kCellMinb) cell_kernel(const StageArgs<double> a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = row_block() * blockDim.y + threadIdx.y;
    if (i >= a.nx || r >= a.ny * (a.k1 - a.k0)) return;
    const int j = r % a.ny, k = r / a.ny + a.k0;
    cell_compute<double, PHYS, IS3D, true>(a, i + 2, j + 2, k + 2);
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

template <int PHYS, bool EXACT>
cudaError_t flux_x_launch(const StageArgs<double> &a, cudaStream_t stream) {
    const int strips = flux_x_strips(a.nx, a.ny, a.k1 - a.k0);
    flux_x_kernel<PHYS, EXACT><<<(strips + 3) / 4, kSplitThreads, 0, stream>>>(a, strips);
    return cudaGetLastError();
}

template <int PHYS, bool EXACT, int DIR>
cudaError_t flux_march_launch(const StageArgs<double> &a, cudaStream_t stream) {
    constexpr size_t smem = kSplitThreads / 32 * kMarchDoubles<PHYS> * sizeof(double);
    auto kernel = flux_march_kernel<PHYS, DIR, EXACT>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int n = DIR == 1 ? a.ny : a.k1 - a.k0;
    const int strips = march_strips(DIR == 1 ? a.nx * (a.k1 - a.k0) : a.nx * a.ny);
    const int seg = march_segment(n, [&](int len) { return (long long)strips * ((n + len - 1) / len); });
    const int warps = strips * ((n + seg - 1) / seg);
    kernel<<<(warps + 3) / 4, kSplitThreads, smem, stream>>>(a, strips, seg);
    return cudaGetLastError();
}

template <int PHYS, bool IS3D>
cudaError_t cell_launch(const StageArgs<double> &a, const KindConfig &c, cudaStream_t stream) {
    const dim3 block(c.bx, c.by), grid = row_grid(a.nx, (long long)a.ny * (a.k1 - a.k0), c.bx, c.by);
    cell_kernel<PHYS, IS3D><<<grid, block, 0, stream>>>(a);
    return cudaGetLastError();
}

template <int PHYS, bool EXACT>
cudaError_t split_kind_dispatch(const StageArgs<double> &a, int kind, const KindConfig &c, cudaStream_t stream) {
    if (a.k0 < 0 || a.k1 > a.nz || a.k0 > a.k1) return cudaErrorInvalidValue;
    if (a.k0 == a.k1) return cudaSuccess;  // no planes
    switch (kind) {
    case kFaceX: return flux_x_launch<PHYS, EXACT>(a, stream);
    case kFaceY: return flux_march_launch<PHYS, EXACT, 1>(a, stream);
    case kFaceZ: return a.nz > 1 ? flux_march_launch<PHYS, EXACT, 2>(a, stream) : cudaSuccess;
    case kCell: return a.nz > 1 ? cell_launch<PHYS, true>(a, c, stream) : cell_launch<PHYS, false>(a, c, stream);
    default: return cudaErrorInvalidValue;
    }
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
cudaError_t launch_split_kind(const StageArgs<S> &a, int physics, bool exact, int kind, const KindConfig &c,
                              cudaStream_t stream) {
    if (!valid_kind_config(kind, c)) return cudaErrorInvalidValue;
    switch (physics) {
    case kIdeal:
        return exact ? split_kind_dispatch<kIdeal, true>(a, kind, c, stream)
                     : split_kind_dispatch<kIdeal, false>(a, kind, c, stream);
    case kPimunu:
        return exact ? split_kind_dispatch<kPimunu, true>(a, kind, c, stream)
                     : split_kind_dispatch<kPimunu, false>(a, kind, c, stream);
    case kPimunuPi:
        return exact ? split_kind_dispatch<kPimunuPi, true>(a, kind, c, stream)
                     : split_kind_dispatch<kPimunuPi, false>(a, kind, c, stream);
    default: return cudaErrorInvalidValue;
    }
}

template <typename S>
cudaError_t launch_stage_split(const StageArgs<S> &a, int physics, bool exact, const SplitConfig &c,
                               cudaStream_t stream) {
    for (int kind = 0; kind < kNumSplitKinds; ++kind) {
        const cudaError_t e = launch_split_kind<S>(a, physics, exact, kind, c.k[kind], stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <typename S>
cudaError_t launch_stage_split(const StageArgs<S> &a, int physics, bool exact, cudaStream_t stream) {
    return launch_stage_split<S>(a, physics, exact, default_split_config(), stream);
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

// The set-up launches and the validity diagnostics serve both storage types;
// the stage launches are FP64 (the FP32 form has the tile kernel).
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
#define VAH_INSTANTIATE_STAGE(S)                                                                                \
    template cudaError_t launch_stage<S>(const StageArgs<S> &, int, cudaStream_t);                              \
    template cudaError_t launch_split_kind<S>(const StageArgs<S> &, int, bool, int, const KindConfig &,         \
                                              cudaStream_t);                                                    \
    template cudaError_t launch_stage_split<S>(const StageArgs<S> &, int, bool, const SplitConfig &,            \
                                               cudaStream_t);                                                   \
    template cudaError_t launch_stage_split<S>(const StageArgs<S> &, int, bool, cudaStream_t);

}  // namespace vah
