// vah_march.cuh -- the flux differences of an RK stage (FP64): each face is
// evaluated once, each cell's limited slope along an axis is formed once, and
// one value per field, axis and cell leaves the launch.
//
// One thread per face (four loads per field, both slopes, both evaluations
// stored) moved 96 values per cell and stage through HBM and held 32 states in
// registers at 16 warps per SM, where load latency was the bound. Here a
// face's fields are split over two lanes, l and l ^ 16, eight each: half the
// registers per thread, so 20 and more warps per SM. The lanes exchange what
// the inversions need (six values per state), the lower lane finds the right
// state's root and the upper lane the left one's, and they exchange the two
// velocities.
//   flux_x: 16 consecutive cells of the plane's rows (ghost cells included, so
//     that rows of any length pack), each lane pair its cell's two edge states
//     from three loads; the neighbour's edge state and the -1/2 flux come
//     through shuffles. Cells 1 to 14 of the 16 are owned.
//   flux_march: 16 columns, walked in segments along y or eta; the last two
//     values, the left state and the lower face's flux of each field wait in
//     shared memory (512 bytes per column), the next value is loaded a step
//     ahead. A segment's first face is its start-up (one in seg + 1).
// Each writes H(-1/2) - H(+1/2) as the cell evaluates the two faces, which the
// cell launch reads.
#pragma once

#include "vah_stage.cuh"

namespace vah {

// 4 times the limited half slope of approx_derivative: the edge states of a
// cell are q -+ limited4 / 4, bit for bit q -+ 0.5 approx_derivative. dl, dr:
// the differences to either neighbour, cc = the neighbours' difference. With
// m = min(|dl|, |dr|), slope = min(1.1 m, |cc| / 2) = min(2.2 m, |cc|) / 2.
// The minima compare bit patterns (non-negative doubles order like integers,
// NaNs above all, so a NaN is passed over as fmin does) and the signs are bit
// tests: integer work beside a busy FP64 pipe.
VAH_HD double limited4(double dl, double dr, double cc) {
#ifdef __CUDA_ARCH__
    constexpr unsigned long long kAbs = 0x7fffffffffffffffull;
    const unsigned long long bl = (unsigned long long)__double_as_longlong(dl), br = (unsigned long long)__double_as_longlong(dr);
    const unsigned long long m = min(bl & kAbs, br & kAbs);
    const double m22 = 2.2 * __longlong_as_double((long long)m);
    unsigned long long r = min((unsigned long long)__double_as_longlong(m22), (unsigned long long)__double_as_longlong(cc) & kAbs);
    r |= bl & ~kAbs;
    return (long long)(bl ^ br) < 0 ? 0.0 : __longlong_as_double((long long)r);
#else
    const double m = fmin(2.2 * fmin(fabs(dl), fabs(dr)), fabs(cc));
    const bool neg = dl < 0.0;
    return neg == (dr < 0.0) ? (neg ? -m : m) : 0.0;
#endif
}

// Strips of flux_x over nk planes: 14 owned cells each of the planes' interior
// rows (ghost cells included) laid end to end.
VAH_HD int flux_x_strips(int nx, int ny, int nk) { return (int)(((long long)nk * ny * (nx + 4) + 9) / 14); }

// Strips of flux_march: 16 columns across the axis each.
VAH_HD int march_strips(int columns) { return (columns + 15) / 16; }

// The fields of the lower (0) and upper (1) lane of a pair, the inversion's
// inputs first: T^{tau tau}, T^{tau x}, T^{tau y} with their pi, and
// T^{tau eta} with its pi, P_L, Pi. An odd count repeats the last field.
template <int PHYS>
struct Halves {
    static constexpr int N = Phys<PHYS>::PIMUNU ? 8 : 3;
    VAH_HD static constexpr int field(int half, int k) {
        constexpr int ideal[2][8] = {{0, 1, 2}, {3, 4, 4}};
        constexpr int shear[2][8] = {{0, 5, 1, 6, 2, 7, 9, 10}, {3, 8, 4, 11, 12, 13, 14, 14}};
        constexpr int bulk[2][8] = {{0, 5, 1, 6, 2, 7, 9, 10}, {3, 8, 4, 15, 11, 12, 13, 14}};
        return PHYS == kIdeal ? ideal[half][k] : (PHYS == kPimunu ? shear[half][k] : bulk[half][k]);
    }
};

// Shared memory of one warp of flux_march, in doubles: two q values, the left
// state and the lower face's flux per field and column.
template <int PHYS>
constexpr int kMarchDoubles = 5 * Halves<PHYS>::N * 32;

#ifdef __CUDACC__

constexpr unsigned kFullWarp = 0xffffffffu;

// The field pointers of a lane's half, from a table in shared memory (one per
// block: read where they are used, so that they hold no registers through the
// solves) ...
struct HalfPointers {
    const double *q_[8][2];
    double *D_[3][8][2];
    __device__ __forceinline__ const double *q(int n, int half) const { return q_[n][half]; }
    __device__ __forceinline__ double *D(int d, int n, int half) const { return D_[d][n][half]; }
};
// ... or selected from the launch's parameters. flux_x is faster with the
// table (104 against 119 us on the 121x121x81 event: 96 registers without
// spills), flux_march with the selection (104 against 112 us along y: it has
// the registers, and its copies' addresses do not wait for a table read).
template <int PHYS>
struct HalfSelect {
    const StageArgs<double> &a;
    __device__ __forceinline__ const double *q(int n, int half) const {
        return half ? a.qin[Halves<PHYS>::field(1, n)] : a.qin[Halves<PHYS>::field(0, n)];
    }
    __device__ __forceinline__ double *D(int d, int n, int half) const {
        return half ? a.D[d][Halves<PHYS>::field(1, n)] : a.D[d][Halves<PHYS>::field(0, n)];
    }
};
// By one thread each (id 0 to 15) of the block; a barrier before use.
template <int PHYS>
__device__ __forceinline__ void set_half_pointers(HalfPointers &h, const StageArgs<double> &a, int id) {
    const int half = id & 1, k = id >> 1;
    if (id >= 2 * Halves<PHYS>::N) return;
    int n = 0;
#pragma unroll
    for (int j = 0; j < Halves<PHYS>::N; ++j)
        if (j == k) n = half ? Halves<PHYS>::field(1, j) : Halves<PHYS>::field(0, j);
    h.q_[k][half] = a.qin[n];
    for (int d = 0; d < 3; ++d) h.D_[d][k][half] = a.D[d][n];
}

// An 8-byte asynchronous copy into shared memory, and the wait for all of a thread's.
__device__ __forceinline__ void copy8_async(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ Guess guess_at(const StageArgs<double> &a, int s) {
    return newton_guess(ldg(a.uin[1] + s), ldg(a.uin[2] + s));
}

// A lane's share of a state's inversion inputs: (m0, m1, m2) or (m3, P_L, Pi).
struct Share {
    double a, b, c;
};
template <int PHYS>
__device__ __forceinline__ Share inv_share(const double *x, int half) {
    if (!Phys<PHYS>::PIMUNU) return {x[0], x[1], half ? 0.0 : x[2]};
    return {x[0] - x[1], half ? x[2] : x[2] - x[3], half ? (Phys<PHYS>::BULK ? x[3] : 0.0) : x[4] - x[5]};
}

// The weights of a face's evaluations by its left cell (s) and its right cell
// (s + st): H = wR qR + wL qL each; equal where every iteration reaches its
// root, which is nearly everywhere (else differ is true for the whole warp).
// qR, qL: this lane's fields of the two states.
struct FaceWeights {
    double wRl, wLl, wRr, wLr;
    int fails_l, fails_r;  // this lane's state: the evaluation's status
    bool differ;
};
template <int PHYS>
__device__ __forceinline__ void face_weights_pair(const StageArgs<double> &a, int half, int s, int st, int dir,
                                                  const double *qR, const double *qL, const Guess &gl, const Guess &gr,
                                                  bool need_l, bool need_r, FaceWeights &w) {
    const Share R = inv_share<PHYS>(qR, half), L = inv_share<PHYS>(qL, half);
    const Share keep = half ? L : R, give = half ? R : L;
    const Share got = {__shfl_xor_sync(kFullWarp, give.a, 16), __shfl_xor_sync(kFullWarp, give.b, 16),
                       __shfl_xor_sync(kFullWarp, give.c, 16)};
    const Share lo = half ? got : keep, hi = half ? keep : got;
    const InvIn q = {lo.a, lo.b, lo.c, hi.a, hi.b, hi.c};  // lower lane: the right state, upper lane: the left
    InvRoot r;
    invert_root(a.t_src, q, r);
    const double v = root_velocity(r, dir == 1 ? q.m2 : q.m1, dir);
    const bool bad_l = need_l && !newton_reaches(r, gl), bad_r = need_r && !newton_reaches(r, gr);
    w.fails_l = w.fails_r = 0;
    w.differ = __any_sync(kFullWarp, bad_l || bad_r);
    if (!w.differ) {
        const double o = __shfl_xor_sync(kFullWarp, v, 16);
        face_weights_of(half ? o : v, half ? v : o, w.wRl, w.wLl);
        w.wRr = w.wRl;
        w.wLr = w.wLl;
        return;
    }
    double vl = v, vr = v;
    if (bad_l)
        w.fails_l = face_velocity_iterated<false>(a.t_src, q, dir, ldg(a.ein + s), ldg(a.uin[1] + s), ldg(a.uin[2] + s), &vl);
    if (bad_r)
        w.fails_r = face_velocity_iterated<false>(a.t_src, q, dir, ldg(a.ein + s + st), ldg(a.uin[1] + s + st),
                                                  ldg(a.uin[2] + s + st), &vr);
    __syncwarp();
    const double ol = __shfl_xor_sync(kFullWarp, vl, 16), orr = __shfl_xor_sync(kFullWarp, vr, 16);
    face_weights_of(half ? ol : vl, half ? vl : ol, w.wRl, w.wLl);
    face_weights_of(half ? orr : vr, half ? vr : orr, w.wRr, w.wLr);
}

// One state's status of one evaluation into [face fallbacks, -, NaNs].
__device__ __forceinline__ void count_status(unsigned long long *counters, int status) {
    if (!counters || status == 0) return;
    atomicAdd(counters + 0, 1ull);
    if (status == 2) atomicAdd(counters + 2, 1ull);
}

template <int PHYS, bool EXACT>
__device__ __forceinline__ void flux_x(const StageArgs<double> &a, const HalfPointers &hp, int strip) {
    constexpr int N = Halves<PHYS>::N;
    const int half = (threadIdx.x >> 4) & 1, pos = threadIdx.x & 15;
    const int rows = a.ny * a.ncx, total = rows * (a.k1 - a.k0), want = 14 * strip + 1 + pos;
    const int f = min(want, total - 1);
    const int k = f / rows, rem = f - k * rows, i = rem % a.ncx;
    const int s = rem + 2 * a.ncx + (int)a.plane * (a.k0 + 2 + k);
    double qR[N], qL[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const double *q = hp.q(n, half) + s;
        const double qm = ldg(q - 1), q0 = ldg(q), qp = ldg(q + 1);
        const double m = limited4(q0 - qm, qp - q0, qp - qm);
        qL[n] = fma(0.25, m, q0);
        qR[n] = __shfl_down_sync(kFullWarp, fma(-0.25, m, q0), 1, 16);
    }
    const Guess gl = guess_at(a, s);
    const Guess gr = {__shfl_down_sync(kFullWarp, gl.v0, 1, 16), __shfl_down_sync(kFullWarp, gl.r2, 1, 16)};
    const bool face = pos < 15 && want < total;  // position 15 has no right state
    const bool need_l = face && i >= (EXACT ? 2 : 1) && i <= a.nx + 1, need_r = EXACT && face && i >= 1 && i <= a.nx;
    FaceWeights w;
    face_weights_pair<PHYS>(a, half, s, 1, 0, qR, qL, gl, gr, need_l, need_r, w);
    const bool own = pos >= 1 && face && i >= 2 && i <= a.nx + 1;
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const double h = fma(w.wRl, qR[n], w.wLl * qL[n]);
        double hr = h;
        if (EXACT && w.differ) hr = fma(w.wRr, qR[n], w.wLr * qL[n]);
        const double hm = __shfl_up_sync(kFullWarp, hr, 1, 16);
        if (own) hp.D(0, n, half)[s] = hm - h;
    }
    if (w.differ) {
        // an evaluation counts once, in the warp that owns its cell (shared faces: their left cell, or the row's first)
        if (need_l && (pos >= 1 || strip == 0)) count_status(a.counters, w.fails_l);
        if (need_r && pos <= 13) count_status(a.counters, w.fails_r);
    }
}

// Columns [16 strip, +16) of the lattice across DIR (1: y, 2: eta), cells
// [m0, m1) along it (interior indices). sm: this warp's shared memory.
template <int PHYS, int DIR, bool EXACT, typename Pointers>
__device__ __forceinline__ void flux_march(const StageArgs<double> &a, const Pointers &hp, int strip, int m0, int m1,
                                           double *sm) {
    constexpr int N = Halves<PHYS>::N;
    const int lane = threadIdx.x & 31, half = lane >> 4, pos = lane & 15;
    const int columns = DIR == 1 ? a.nx * (a.k1 - a.k0) : a.nx * a.ny, plane = (int)a.plane;
    const bool live = 16 * strip + pos < columns;
    const int f = min(16 * strip + pos, columns - 1), outer = f / a.nx, i = f - outer * a.nx;
    const int st = DIR == 1 ? a.ncx : plane;
    const int base = i + 2 + (DIR == 1 ? plane * (a.k0 + 2 + outer) : a.ncx * (outer + 2));
    double *Q = sm + lane, *QL = Q + 3 * N * 32, *HR = QL + N * 32;  // [3][N][32], [N][32], [N][32]
    int s = base + st * (m0 + 1);  // the left cell of the segment's first face
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const double *q = hp.q(n, half) + s;
        const double qm = ldg(q - st), q0 = ldg(q), qp = ldg(q + st);
        copy8_async(Q + (2 * N + n) * 32, q + 2 * st);
        QL[n * 32] = fma(0.25, limited4(q0 - qm, qp - q0, qp - qm), q0);
        Q[n * 32] = q0;
        Q[(N + n) * 32] = qp;
    }
    Guess gl = guess_at(a, s);
    double un1 = ldg(a.uin[1] + s + st), un2 = ldg(a.uin[2] + s + st);  // the right cell's velocity
    double *Q0 = Q, *Q1 = Q + N * 32, *Q2 = Q1 + N * 32;  // q of the left cell, the right one and the next
#pragma unroll 1
    for (int m = m0 - 1; m < m1; ++m, s += st) {  // the face at +1/2 of cell m
        double qR[N], qL[N];
        copies_wait();
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const double q0 = Q0[n * 32], q1 = Q1[n * 32], v = Q2[n * 32];
            const double l = limited4(q1 - q0, v - q1, v - q0);
            qL[n] = QL[n * 32];
            qR[n] = fma(-0.25, l, q1);
            QL[n * 32] = fma(0.25, l, q1);
        }
        double *const free_row = Q0;
        Q0 = Q1;
        Q1 = Q2;
        Q2 = free_row;
        const Guess gr = newton_guess(un1, un2);
        if (m + 1 < m1) {
#pragma unroll
            for (int n = 0; n < N; ++n) copy8_async(Q2 + n * 32, hp.q(n, half) + s + 3 * st);
            un1 = ldg(a.uin[1] + s + 2 * st);
            un2 = ldg(a.uin[2] + s + 2 * st);
        }
        const bool mine = m >= m0;  // cell m belongs to this segment
        const bool need_l = EXACT ? mine : true, need_r = EXACT && m + 1 < m1;
        FaceWeights w;
        face_weights_pair<PHYS>(a, half, s, st, DIR, qR, qL, gl, gr, need_l, need_r, w);
        gl = gr;
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const double h = fma(w.wRl, qR[n], w.wLl * qL[n]);
            double hr = h;
            if (EXACT && w.differ) hr = fma(w.wRr, qR[n], w.wLr * qL[n]);
            if (mine && live) hp.D(DIR, n, half)[s] = HR[n * 32] - h;
            HR[n * 32] = hr;
        }
        if (w.differ && live) {
            // shared faces: the lattice's first face has no owner but the segment that starts there
            if (EXACT ? need_l : (mine || m == -1)) count_status(a.counters, w.fails_l);
            if (need_r) count_status(a.counters, w.fails_r);
        }
    }
}

#endif  // __CUDACC__

}  // namespace vah
