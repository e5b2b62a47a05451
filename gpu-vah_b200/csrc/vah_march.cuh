// vah_march.cuh -- the flux differences of an RK stage: each face is evaluated
// once, each cell's limited slope along an axis is formed once, and
// one value per field, axis and cell leaves the launch.
//
// One thread per face (four loads per field, both slopes, both evaluations
// stored) moved 96 values per cell and stage through HBM and held 32 states in
// registers at 16 warps per SM, where load latency was the bound. Here (W
// columns per warp):
//   flux_x: W consecutive cells of the plane's rows (ghost cells included, so
//     that rows of any length pack), each its two edge states from three loads;
//     the neighbour's edge state and the -1/2 flux come through shuffles. The
//     cells 1 to W - 2 are owned.
//   flux_march: W columns, walked in segments along y or eta; the last two
//     values, the left state and the lower face's flux of each field wait in
//     shared memory, the next value is copied in a step ahead. A segment's
//     first face is its start-up (one in seg + 1).
// FP64 faces are split over two lanes, l and l ^ 16, eight fields each (W =
// 16): half the registers per thread, so that nothing spills at 16 and more
// warps per SM (the unsplit march spilled at 12: 151 us against 104 along y of
// the 121x121x81 event). The lanes exchange what the inversions need (six
// values per state), the lower lane finds the right state's root and the upper
// lane the left one's, and they exchange the two velocities. FP32 faces fit one
// lane (W = 32); split, their roots' overhead came twice as often (205 us
// against 178 for all axes).
// Each writes H(-1/2) - H(+1/2) as the cell evaluates the two faces, which the
// cell launch reads.
// S: the storage and arithmetic type of states and fluxes (double, or float
// for the FP32 form); the inversions run in FP64 either way.
#pragma once

#include "vah_stage.cuh"

namespace vah {

// 4 times the limited half slope of approx_derivative: the edge states of a
// cell are q -+ limited4 / 4, bit for bit q -+ 0.5 approx_derivative. dl, dr:
// the differences to either neighbour, cc = the neighbours' difference. With
// m = min(|dl|, |dr|), slope = min(1.1 m, |cc| / 2) = min(2.2 m, |cc|) / 2.
// The minima compare bit patterns (non-negative numbers order like integers,
// NaNs above all, so a NaN is passed over as fmin does) and the signs are tests of
// the upper bits, a NaN not being below zero whatever its sign bit (the device's
// own FP64 NaN has it set): integer work beside a busy FP64 pipe.
VAH_HD bool below_zero(uint64_t bits) { return (uint32_t)(bits >> 32) - 0x80000000u <= 0x7ff00000u; }
VAH_HD bool below_zero(uint32_t bits) { return bits - 0x80000000u <= 0x7f800000u; }
template <typename U>
VAH_HD U smaller(U a, U b) { return b < a ? b : a; }

VAH_HD double limited4(double dl, double dr, double cc) {
    constexpr uint64_t kSign = 1ull << 63;
    const uint64_t bl = double_bits(dl), br = double_bits(dr);
    const double m22 = 2.2 * bits_double(smaller(bl & ~kSign, br & ~kSign));
    const uint64_t r = smaller(double_bits(m22), double_bits(cc) & ~kSign);
    const bool neg = below_zero(bl);
    return neg != below_zero(br) ? 0.0 : bits_double(r | (neg ? kSign : 0));
}
// The same in FP32.
VAH_HD float limited4(float dl, float dr, float cc) {
    constexpr uint32_t kSign = 1u << 31;
    const uint32_t bl = float_bits(dl), br = float_bits(dr);
    const float m22 = 2.2f * bits_float(smaller(bl & ~kSign, br & ~kSign));
    const uint32_t r = smaller(float_bits(m22), float_bits(cc) & ~kSign);
    const bool neg = below_zero(bl);
    return neg != below_zero(br) ? 0.0f : bits_float(r | (neg ? kSign : 0));
}

// The lanes' shares of a face: whether two lanes split its fields, the columns
// W per warp, the fields N per lane and which they are. Split: the inversion's
// inputs first, T^{tau tau}, T^{tau x}, T^{tau y} with their pi in the lower
// lane (0), T^{tau eta} with its pi, P_L, Pi in the upper (1); an odd count
// repeats the last field.
template <typename S, int PHYS>
struct Lanes {
    static constexpr bool SPLIT = sizeof(S) == 8;
    static constexpr int W = SPLIT ? 16 : 32;
    static constexpr int N = !SPLIT ? Phys<PHYS>::NQ : (Phys<PHYS>::PIMUNU ? 8 : 3);
    VAH_HD static constexpr int field(int half, int k) {
        constexpr int ideal[2][8] = {{0, 1, 2}, {3, 4, 4}};
        constexpr int shear[2][8] = {{0, 5, 1, 6, 2, 7, 9, 10}, {3, 8, 4, 11, 12, 13, 14, 14}};
        constexpr int bulk[2][8] = {{0, 5, 1, 6, 2, 7, 9, 10}, {3, 8, 4, 15, 11, 12, 13, 14}};
        if (!SPLIT) return k;
        return PHYS == kIdeal ? ideal[half][k] : (PHYS == kPimunu ? shear[half][k] : bulk[half][k]);
    }
};

// Strips of flux_x over nk planes: W - 2 owned cells each of the planes'
// interior rows (ghost cells included) laid end to end; the first and last
// owned cells of the run are its third and its third last.
template <typename S>
VAH_HD int flux_x_strips(int nx, int ny, int nk) {
    constexpr int own = Lanes<S, 0>::W - 2;
    return (int)(((long long)nk * ny * (nx + 4) - 4 + own - 1) / own);
}

// Strips of flux_march: W columns across the axis each.
template <typename S>
VAH_HD int march_strips(int columns) {
    return (columns + Lanes<S, 0>::W - 1) / Lanes<S, 0>::W;
}

// Shared memory of one warp of flux_march, in values: three q values, the left
// state and the lower face's flux per field and column.
template <typename S, int PHYS>
constexpr int kMarchValues = 5 * Lanes<S, PHYS>::N * 32;

#ifdef __CUDACC__

constexpr unsigned kFullWarp = 0xffffffffu;

// The field pointers of a lane's share, selected from the launch's parameters ...
template <typename S, int PHYS>
struct SelectPointers {
    const StageArgs<S> &a;
    using L = Lanes<S, PHYS>;
    __device__ __forceinline__ const S *q(int n, int half) const {
        return half ? a.qin[L::field(1, n)] : a.qin[L::field(0, n)];
    }
    __device__ __forceinline__ S *D(int d, int n, int half) const {
        return half ? a.D[d][L::field(1, n)] : a.D[d][L::field(0, n)];
    }
};
// ... or from a table in shared memory, one per block: read where they are
// used, they hold no registers through the solves. FP64's flux_x is faster with
// the table (104 against 119 us on the 121x121x81 event), flux_march with the
// selection (104 against 112 us along y: its copies' addresses do not wait for
// a table read). The batches, whose arguments are in memory anyway, use it
// throughout.
template <typename S>
struct TablePointers {
    const S *q_[16][2];
    S *D_[3][16][2];
    __device__ __forceinline__ const S *q(int n, int half) const { return q_[n][half]; }
    __device__ __forceinline__ S *D(int d, int n, int half) const { return D_[d][n][half]; }
};
// By one thread each (id 0 to 31) of the block; a barrier before use.
template <int PHYS, typename S>
__device__ __forceinline__ void set_table_pointers(TablePointers<S> &h, const StageArgs<S> &a, int id) {
    using L = Lanes<S, PHYS>;
    const int half = id & 1, k = id >> 1;
    if (id >= 2 * L::N) return;
    int n = 0;
#pragma unroll
    for (int j = 0; j < L::N; ++j)
        if (j == k) n = half ? L::field(1, j) : L::field(0, j);
    h.q_[k][half] = a.qin[n];
    for (int d = 0; d < 3; ++d) h.D_[d][k][half] = a.D[d][n];
}

// One value's asynchronous copy into shared memory, and the wait for all of a thread's.
template <typename S>
__device__ __forceinline__ void copy_async(S *dst, const S *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(S))
                 : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <typename S>
__device__ __forceinline__ Guess guess_at(const StageArgs<S> &a, int s) {
    return newton_guess((double)load(a.uin[1] + s), (double)load(a.uin[2] + s));
}
__device__ __forceinline__ double fma_(double x, double y, double z) { return fma(x, y, z); }
__device__ __forceinline__ float fma_(float x, float y, float z) { return fmaf(x, y, z); }

// A lane's share of a state's inversion inputs: (m0, m1, m2) or (m3, P_L, Pi).
struct Share {
    double a, b, c;
};
template <int PHYS, typename S>
__device__ __forceinline__ Share inv_share(const S *q, int half) {
    double x[6];
#pragma unroll
    for (int n = 0; n < (Phys<PHYS>::PIMUNU ? 6 : 3); ++n) x[n] = (double)q[n];
    if (!Phys<PHYS>::PIMUNU) return {x[0], x[1], half ? 0.0 : x[2]};
    return {x[0] - x[1], half ? x[2] : x[2] - x[3], half ? (Phys<PHYS>::BULK ? x[3] : 0.0) : x[4] - x[5]};
}

// The weights of a face's evaluations by its left cell (s) and its right cell
// (s + st): H = wR qR + wL qL each; equal where every iteration reaches its
// root, which is nearly everywhere (else differ is true for the whole warp).
template <typename S>
struct FaceWeights {
    S wRl, wLl, wRr, wLr;
    int fails_l, fails_r;  // the evaluations' inversions that fell back in this lane; bit 8: a NaN
    bool differ;
};
template <typename S>
__device__ __forceinline__ void set_weights(double vR, double vL, S &wR, S &wL) {
    double r, l;
    face_weights_of(vR, vL, r, l);
    wR = (S)r;
    wL = (S)l;
}
// One state's velocity as the cell at s evaluates it, by the iteration.
template <typename S>
__device__ __forceinline__ int velocity_at(const StageArgs<S> &a, const InvIn &q, int dir, int s, double *v) {
    const int st = face_velocity_iterated<sizeof(S) == 4>(a.t_src, q, dir, (double)load(a.ein + s),
                                                          (double)load(a.uin[1] + s), (double)load(a.uin[2] + s), v);
    return (st != 0) + (st == 2 ? 256 : 0);
}

// qR, qL: this lane's fields of the two states.
template <int PHYS, typename S>
__device__ __forceinline__ void face_weights_lanes(const StageArgs<S> &a, int half, int s, int st, int dir, const S *qR,
                                                   const S *qL, const Guess &gl, const Guess &gr, bool need_l,
                                                   bool need_r, FaceWeights<S> &w) {
    constexpr bool FAST = sizeof(S) == 4;
    w.fails_l = w.fails_r = 0;
    if constexpr (Lanes<S, PHYS>::SPLIT) {
        const Share R = inv_share<PHYS>(qR, half), L = inv_share<PHYS>(qL, half);
        const Share keep = half ? L : R, give = half ? R : L;
        const Share got = {__shfl_xor_sync(kFullWarp, give.a, 16), __shfl_xor_sync(kFullWarp, give.b, 16),
                           __shfl_xor_sync(kFullWarp, give.c, 16)};
        const Share lo = half ? got : keep, hi = half ? keep : got;
        const InvIn q = {lo.a, lo.b, lo.c, hi.a, hi.b, hi.c};  // lower lane: the right state, upper lane: the left
        InvRoot r;
        invert_root<FAST>(a.t_src, q, r);
        const double v = root_velocity(r, dir == 1 ? q.m2 : q.m1, dir);
        const bool bad_l = need_l && !newton_reaches(r, gl), bad_r = need_r && !newton_reaches(r, gr);
        w.differ = __any_sync(kFullWarp, bad_l || bad_r);
        if (!w.differ) {
            const double o = __shfl_xor_sync(kFullWarp, v, 16);
            set_weights(half ? o : v, half ? v : o, w.wRl, w.wLl);
            w.wRr = w.wRl;
            w.wLr = w.wLl;
            return;
        }
        double vl = v, vr = v;
        if (bad_l) w.fails_l = velocity_at(a, q, dir, s, &vl);
        if (bad_r) w.fails_r = velocity_at(a, q, dir, s + st, &vr);
        __syncwarp();
        const double ol = __shfl_xor_sync(kFullWarp, vl, 16), orr = __shfl_xor_sync(kFullWarp, vr, 16);
        set_weights(half ? ol : vl, half ? vl : ol, w.wRl, w.wLl);
        set_weights(half ? orr : vr, half ? vr : orr, w.wRr, w.wLr);
    } else {
        double dR[16], dL[16];
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            dR[n] = n < Phys<PHYS>::NQ ? (double)qR[n] : 0.0;
            dL[n] = n < Phys<PHYS>::NQ ? (double)qL[n] : 0.0;
        }
        FaceRoots f;
        face_roots<PHYS, FAST>(a.t_src, dR, dL, f);
        const double vR = root_velocity(f.R, dir == 1 ? f.qR.m2 : f.qR.m1, dir);
        const double vL = root_velocity(f.L, dir == 1 ? f.qL.m2 : f.qL.m1, dir);
        const bool rl = need_l && !newton_reaches(f.R, gl), ll = need_l && !newton_reaches(f.L, gl);
        const bool rr = need_r && !newton_reaches(f.R, gr), lr = need_r && !newton_reaches(f.L, gr);
        w.differ = __any_sync(kFullWarp, rl || ll || rr || lr);
        set_weights(vR, vL, w.wRl, w.wLl);
        w.wRr = w.wRl;
        w.wLr = w.wLl;
        if (!w.differ) return;
        double vRl = vR, vLl = vL, vRr = vR, vLr = vL;
        if (rl) w.fails_l = velocity_at(a, f.qR, dir, s, &vRl);
        if (ll) w.fails_l += velocity_at(a, f.qL, dir, s, &vLl);
        if (rr) w.fails_r = velocity_at(a, f.qR, dir, s + st, &vRr);
        if (lr) w.fails_r += velocity_at(a, f.qL, dir, s + st, &vLr);
        set_weights(vRl, vLl, w.wRl, w.wLl);
        set_weights(vRr, vLr, w.wRr, w.wLr);
        __syncwarp();
    }
}

// One evaluation's fallbacks into the counters [face fallbacks, -, NaNs].
__device__ __forceinline__ void count_fails(unsigned long long *counters, int fails) {
    if (!counters || fails == 0) return;
    atomicAdd(counters + 0, (unsigned long long)(fails & 255));
    if (fails >> 8) atomicAdd(counters + 2, 1ull);
}

template <int PHYS, bool EXACT, typename S, typename Pointers>
__device__ __forceinline__ void flux_x(const StageArgs<S> &a, const Pointers &hp, int strip) {
    constexpr int N = Lanes<S, PHYS>::N, W = Lanes<S, PHYS>::W;
    const int half = W == 16 ? (threadIdx.x >> 4) & 1 : 0, pos = threadIdx.x & (W - 1);
    const int rows = a.ny * a.ncx, total = rows * (a.k1 - a.k0), want = (W - 2) * strip + 1 + pos;
    const int f = min(want, total - 1);
    const int k = f / rows, rem = f - k * rows, i = rem % a.ncx;
    const int s = rem + 2 * a.ncx + (int)a.plane * (a.k0 + 2 + k);
    S qR[N], qL[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const S *q = hp.q(n, half) + s;
        const S qm = load(q - 1), q0 = load(q), qp = load(q + 1);
        const S m = limited4(q0 - qm, qp - q0, qp - qm);
        qL[n] = fma_(S(0.25), m, q0);
        qR[n] = __shfl_down_sync(kFullWarp, fma_(S(-0.25), m, q0), 1, W);
    }
    const Guess gl = guess_at(a, s);
    const Guess gr = {__shfl_down_sync(kFullWarp, gl.v0, 1, W), __shfl_down_sync(kFullWarp, gl.r2, 1, W)};
    const bool face = pos < W - 1 && want < total;  // the last position has no right state
    const bool need_l = face && i >= (EXACT ? 2 : 1) && i <= a.nx + 1, need_r = EXACT && face && i >= 1 && i <= a.nx;
    FaceWeights<S> w;
    face_weights_lanes<PHYS>(a, half, s, 1, 0, qR, qL, gl, gr, need_l, need_r, w);
    const bool own = pos >= 1 && face && i >= 2 && i <= a.nx + 1;
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const S h = fma_(w.wRl, qR[n], w.wLl * qL[n]);
        S hr = h;
        if (EXACT && w.differ) hr = fma_(w.wRr, qR[n], w.wLr * qL[n]);
        const S hm = __shfl_up_sync(kFullWarp, hr, 1, W);
        if (own) hp.D(0, n, half)[s] = hm - h;
    }
    if (w.differ) {
        // an evaluation counts once, in the warp that owns its cell (shared faces: their left cell, or the row's first)
        if (need_l && (pos >= 1 || strip == 0)) count_fails(a.counters, w.fails_l);
        if (need_r && pos <= W - 3) count_fails(a.counters, w.fails_r);
    }
}

// Columns [W strip, +W) of the lattice across DIR (1: y, 2: eta), cells
// [m0, m1) along it (interior indices). sm: this warp's shared memory.
template <int PHYS, int DIR, bool EXACT, typename S, typename Pointers>
__device__ __forceinline__ void flux_march(const StageArgs<S> &a, const Pointers &hp, int strip, int m0, int m1, S *sm) {
    constexpr int N = Lanes<S, PHYS>::N, W = Lanes<S, PHYS>::W;
    const int lane = threadIdx.x & 31, half = W == 16 ? lane >> 4 : 0, pos = lane & (W - 1);
    const int columns = DIR == 1 ? a.nx * (a.k1 - a.k0) : a.nx * a.ny, plane = (int)a.plane;
    const bool live = W * strip + pos < columns;
    const int f = min(W * strip + pos, columns - 1), outer = f / a.nx, i = f - outer * a.nx;
    const int st = DIR == 1 ? a.ncx : plane;
    const int base = i + 2 + (DIR == 1 ? plane * (a.k0 + 2 + outer) : a.ncx * (outer + 2));
    S *Q = sm + lane, *QL = Q + 3 * N * 32, *HR = QL + N * 32;  // [3][N][32], [N][32], [N][32]
    int s = base + st * (m0 + 1);  // the left cell of the segment's first face
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const S *q = hp.q(n, half) + s;
        const S qm = load(q - st), q0 = load(q), qp = load(q + st);
        copy_async(Q + (2 * N + n) * 32, q + 2 * st);
        QL[n * 32] = fma_(S(0.25), limited4(q0 - qm, qp - q0, qp - qm), q0);
        Q[n * 32] = q0;
        Q[(N + n) * 32] = qp;
    }
    Guess gl = guess_at(a, s);
    S un1 = load(a.uin[1] + s + st), un2 = load(a.uin[2] + s + st);  // the right cell's velocity
    S *Q0 = Q, *Q1 = Q + N * 32, *Q2 = Q1 + N * 32;  // q of the left cell, the right one and the next
#pragma unroll 1
    for (int m = m0 - 1; m < m1; ++m, s += st) {  // the face at +1/2 of cell m
        S qR[N], qL[N];
        copies_wait();
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const S q0 = Q0[n * 32], q1 = Q1[n * 32], v = Q2[n * 32];
            const S l = limited4(q1 - q0, v - q1, v - q0);
            qL[n] = QL[n * 32];
            qR[n] = fma_(S(-0.25), l, q1);
            QL[n * 32] = fma_(S(0.25), l, q1);
        }
        S *const free_row = Q0;
        Q0 = Q1;
        Q1 = Q2;
        Q2 = free_row;
        const Guess gr = newton_guess((double)un1, (double)un2);
        if (m + 1 < m1) {
#pragma unroll
            for (int n = 0; n < N; ++n) copy_async(Q2 + n * 32, hp.q(n, half) + s + 3 * st);
            un1 = load(a.uin[1] + s + 2 * st);
            un2 = load(a.uin[2] + s + 2 * st);
        }
        const bool mine = m >= m0;  // cell m belongs to this segment
        const bool need_l = EXACT ? mine : true, need_r = EXACT && m + 1 < m1;
        FaceWeights<S> w;
        face_weights_lanes<PHYS>(a, half, s, st, DIR, qR, qL, gl, gr, need_l, need_r, w);
        gl = gr;
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const S h = fma_(w.wRl, qR[n], w.wLl * qL[n]);
            S hr = h;
            if (EXACT && w.differ) hr = fma_(w.wRr, qR[n], w.wLr * qL[n]);
            if (mine && live) hp.D(DIR, n, half)[s] = HR[n * 32] - h;
            HR[n * 32] = hr;
        }
        if (w.differ && live) {
            // shared faces: the lattice's first face has no owner but the segment that starts there
            if (EXACT ? need_l : (mine || m == -1)) count_fails(a.counters, w.fails_l);
            if (need_r) count_fails(a.counters, w.fails_r);
        }
    }
}

#endif  // __CUDACC__

}  // namespace vah
