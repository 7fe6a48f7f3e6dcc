// Runs of a single grid point (0-D: no propagation) in FP64 with the Cayley
// update: one warp per run, one lane per entry of the density matrix.
//
// What bounds such a run is the latency of a step, and an FP64 instruction
// holds its scheduler's unit for 64 cycles whether one lane or 32 take part
// (measured; see rot_coeffs<double>). The tile kernels give a point to one
// lane, so a 3-level step is about 670 FP64 instructions one after the
// other. With the entry (i, j) of every N x N matrix in lane i N + j a
// product is 4 N of them, and the solve A Y = K runs by Gauss-Jordan
// elimination, which updates all rows of a column at once: about 125 FP64
// instructions (3-level preset, 10,000 steps: 188 -> 51 ms).
// The state in memory, the steps per launch, sources and records are those
// of the tile kernels (cayley_update has the formulas).
#pragma once

#include "tile_kernel.cuh"

namespace mbg {

constexpr int POINT_THREADS = 32;

// 1 / x by two Newton steps from an FP32 reciprocal (21 -> 42 -> 84 bits, the
// last rounded to FP64: the division's result, unless the quotient lies within
// 2^-31 of an ulp of the middle between two numbers): 4 FP64 instructions
// instead of a division's ten. FP32 and back through the bits, because a conversion is
// an FP64 instruction too. x is the squared modulus of a pivot of I + iK,
// whose Hermitian part is I: at least 1; beyond FP32's range the division.
__device__ __forceinline__ double pivot_reciprocal(double x)
{
    const int h = __double2hiint(x);
    if (h < 0x3ff00000 || h >= 0x47000000) return 1.0 / x;  // below 1 (rounding), from 2^113, Inf, NaN
    const float f = __int_as_float(((h - 0x38000000) << 3) | (int) ((unsigned) __double2loint(x) >> 29));
    const int g = __float_as_int(__fdividef(1.0f, f));
    double r = __hiloint2double((g >> 3) + 0x38000000, g << 29);
    r = fma(fma(-x, r, 1.0), r, r);
    return fma(fma(-x, r, 1.0), r, r);
}

template<int N>
__global__ void __launch_bounds__(POINT_THREADS) point_cayley_kernel(const kparams<double> p)
{
    constexpr int NN = N * N;
    constexpr uint32_t ALL = 0xffffffffu;
    static_assert(NN <= 32, "one lane per entry");
    __shared__ tile_lists tl;
    __shared__ src_values<double> sv;
    __shared__ double rho_sh[NN];  // packed, for the record rows
    const tile_desc td = p.tiles[blockIdx.x];
    const run_desc rd = p.runs[td.run];
    const int64_t g0 = (int64_t) rd.offset;
    const uint64_t step0 = *p.step_base + (uint64_t) p.launch_idx * p.depth;
    int nsteps = 0;
    if (step0 < rd.n_t) nsteps = (int) min((uint64_t) p.nsub, (uint64_t) rd.n_t - step0);
    const int lane = threadIdx.x;
    if (lane == 0) gather_lists(p, td, rd, 0, 1, nsteps, tl);

    // lanes beyond the matrix repeat its last entry (and store nothing)
    const int e = min(lane, NN - 1), i = e / N, j = e % N;
    const int m = p.mat[g0];
    const double* cb = p.mc + (uint64_t) (m >= 0 ? m : 0) * p.mstride;
    const pre::cay_layout L = pre::make_cay_layout(N);
    const bool qm = m >= 0 && !is_zero(cb[pre::FD_HAS_QM]);
    // packed index of the entry's real part, its sign of the imaginary part
    const int lo = min(i, j), hi = max(i, j);
    const int q = hi * (hi - 1) / 2 + lo;
    const int at = i == j ? i : N + 2 * q;
    const double sg = i <= j ? 1.0 : -1.0;
    auto entry = [&](int base, double& re, double& im) {
        re = cb[base + at];
        im = i == j ? 0.0 : sg * cb[base + at + 1];
    };
    double hr, hm, mr, mm;  // kappa H0, kappa mu
    entry(L.kH0, hr, hm);
    entry(L.kMu, mr, mm);
    // dissipation half step: c[0 ..] on the populations (diagonal) or c[0] on
    // the entry itself; cim on its imaginary part
    double c[N];
#pragma unroll
    for (int l = 0; l < N; l++)
        c[l] = i == j ? cb[L.dD1 + i * N + l] : l == 0 ? cb[L.dD2 + q] : 0.0;
    const double cim = i == j ? 0.0 : c[0];
    // current: the upper triangle's weights
    const bool mine = lane < NN;
    const double gr = mine && i <= j ? cb[L.gP + at] : 0.0;
    const double gi = mine && i < j ? cb[L.gP + at + 1] : 0.0;
    const double fa = cb[pre::FD_A], fb = cb[pre::FD_BDX], fg = cb[pre::FD_G];

    double E = p.Ein[g0], H = p.Hin[g0], P = p.Pin[g0];
    double xr = p.Din[(uint64_t) at * p.plane + g0];
    double xi = i == j ? 0.0 : sg * p.Din[(uint64_t) (at + 1) * p.plane + g0];

    __syncwarp();
    tile_own<double> own{ 0u, -1, -1, nullptr };
    if (tl.nsrc + tl.nrec > 0 || tl.overflow) {
        prepare_lists<double, POINT_THREADS>(p, tl, sv, step0, nsteps);
        __syncwarp();
        own = own_lists<double, 1>(p, tl, td, 0, nsteps);
    }
    // every lane applies the sources to its copy of E; lane r takes the rows
    // of record r (with more than a tile lists, lane 0 of all)
    const bool rows = own.bits > 255u;  // the same in every lane
    int kind = -1, idx = 0;  // 0 E, 1 P, 2 H, 3 entry idx, 4 inversion, 5 zero; + 8: negated
    uint64_t left = 0;
    double* dst = nullptr;
    if (rows && !tl.overflow && lane < tl.nrec) {
        const rec_desc rc = tl.rec[lane];
        const uint64_t row = tl.row0[lane] + (tl.mask[lane][0] & 1u ? 0u : 1u);
        dst = p.scratch + rc.offset + row;
        left = row < rc.rows ? rc.rows - row : 0;
        kind = rc.type <= 2 || rc.type == 4 ? rc.type : 3;
        if (kind == 3) {
            // populations and coherence parts: an entry of the packed
            // matrix, as in tile_steps
            const uint32_t a = min(rc.row_idx, rc.col_idx), b = max(rc.row_idx, rc.col_idx);
            const uint32_t k = rc.type == 3 ? (a == b ? a : 0xffffffffu)
                                            : N + 2 * (b * (b - 1) / 2 + a) + (rc.type == REC_COH_IM ? 1 : 0);
            if (k < (uint32_t) NN)
                idx = (int) k;
            else
                kind = 5;
            if (rc.type == REC_COH_IM && rc.row_idx > rc.col_idx) kind += 8;
        }
        if (left == 0) kind = -1;  // steps due beyond the last row take none
    }
    auto shf = [&](double v, int src) { return __shfl_sync(ALL, v, src); };
    auto dissipate = [&](double& re, double& im) {
        double s = re;
#pragma unroll
        for (int l = 0; l < N; l++) {
            const double d = shf(re, l * (N + 1));
            s = fma(c[l], i == j ? d : re, s);
        }
        re = s;
        im = fma(cim, im, im);
    };

    for (int t = 0; t < nsteps; t++) {
        const uint64_t n = step0 + (uint64_t) t;
        const uint32_t due = due_records(p, tl, own, t);
        if (m >= 0) E = fma(fa, E, fma(fb, 0.0 - H, -fg * P));
        for_sources(p, rd, tl, sv, own, 0, t, nsteps, n, [&](int jj, int type, double v, double) {
            if (jj == 0 && m >= 0) E = type == 0 ? v : E + v;
        });
        H = 0.0;  // PMC
        if (qm) {
            // A = I + iK, Y = K (K = kappa H0 - E kappa mu)
            double yr = fma(-E, mr, hr), yi = fma(-E, mm, hm);
            double ar = (i == j ? 1.0 : 0.0) - yi, ai = yr;
            double ir = 0.0, ii = 0.0;  // inverse of this row's pivot
#pragma unroll
            for (int k = 0; k < N; k++) {
                const double pr = shf(ar, k * (N + 1)), pi = shf(ai, k * (N + 1));
                const double rk = pivot_reciprocal(fma(pr, pr, pi * pi));
                const double vr = pr * rk, vi = -pi * rk;
                const double kr = shf(ar, k * N + j), ki = shf(ai, k * N + j);
                const double zr = shf(yr, k * N + j), zi = shf(yi, k * N + j);
                const double cr = shf(ar, i * N + k), ci = shf(ai, i * N + k);
                const bool pivot = i == k;
                ir = pivot ? vr : ir;
                ii = pivot ? vi : ii;
                // rows other than k lose their column k
                const double nr = pivot ? 0.0 : -fma(cr, vr, -(ci * vi));
                const double ni = pivot ? 0.0 : -fma(cr, vi, ci * vr);
                if (k + 1 < N) {
                    ar = fma(nr, kr, fma(-ni, ki, ar));
                    ai = fma(nr, ki, fma(ni, kr, ai));
                }
                yr = fma(nr, zr, fma(-ni, zi, yr));
                yi = fma(nr, zi, fma(ni, zr, yi));
            }
            // X = -2i Y
            const double wr = fma(yr, ir, -(yi * ii)), wi = fma(yr, ii, yi * ir);
            const double Xr = wi + wi, Xi = -(wr + wr);
            dissipate(xr, xi);
            // G = X rho1
            double gR = 0.0, gI = 0.0;
#pragma unroll
            for (int l = 0; l < N; l++) {
                const double ur = shf(Xr, i * N + l), ui = shf(Xi, i * N + l);
                const double sr = shf(xr, l * N + j), si = shf(xi, l * N + j);
                gR = fma(ur, sr, fma(-ui, si, gR));
                gI = fma(ur, si, fma(ui, sr, gI));
            }
            // rho2 = rho1 + (G + G^H + G X^H)
            double dr = gR + shf(gR, j * N + i), di = gI - shf(gI, j * N + i);
#pragma unroll
            for (int l = 0; l < N; l++) {
                const double ur = shf(gR, i * N + l), ui = shf(gI, i * N + l);
                const double sr = shf(Xr, j * N + l), si = shf(Xi, j * N + l);
                dr = fma(ur, sr, fma(ui, si, dr));
                di = fma(ui, sr, fma(-ur, si, di));
            }
            xr += dr;
            xi = i == j ? 0.0 : xi + di;
            dissipate(xr, xi);
            // the lower triangle is the upper one's conjugate
            const double tr = shf(xr, lo * N + hi), ti = shf(xi, lo * N + hi);
            xr = tr;
            xi = sg * ti;
            double s = fma(gr, xr, gi * xi);
#pragma unroll
            for (int o = NN <= 16 ? 8 : 16; o > 0; o >>= 1) s += __shfl_xor_sync(ALL, s, o);
            P = shf(s, 0);
        }
        if (rows) {
            if (mine && i <= j) {
                rho_sh[at] = xr;
                if (i < j) rho_sh[at + 1] = xi;
            }
            __syncwarp();
            auto value = [&](int kd, int k) {
                double v = E;
                if (kd == 1) v = P;
                if (kd == 2) v = H;
                if ((kd & 7) == 3) v = rho_sh[k];
                if (kd == 4) v = rho_sh[1] - rho_sh[0];
                if ((kd & 7) == 5) v = 0.0;
                return kd & 8 ? -v : v;
            };
            if (!tl.overflow) {
                if (kind >= 0 && (tl.due[t] >> lane & 1u)) {
                    const double v = value(kind, idx);
                    *dst++ = v;
                    if (--left == 0) kind = -1;
                    if (!isfinite(v)) atomicOr(p.status, STATUS_NONFINITE);
                }
            } else if (lane == 0) {
                for_records(p, rd, tl, own, due, t, n, [](int, int) { return 0.0; },
                    [&](const rec_desc& rc, uint64_t row) {
                        const uint32_t a = min(rc.row_idx, rc.col_idx), b = max(rc.row_idx, rc.col_idx);
                        const uint32_t k = rc.type == 3 ? (a == b ? a : 0xffffffffu)
                                                        : N + 2 * (b * (b - 1) / 2 + a) +
                                (rc.type == REC_COH_IM ? 1 : 0);
                        int kd = rc.type <= 2 || rc.type == 4 ? rc.type : k < (uint32_t) NN ? 3 : 5;
                        if (rc.type == REC_COH_IM && rc.row_idx > rc.col_idx) kd += 8;
                        const double v = value(kd, (kd & 7) == 3 ? (int) k : 0);
                        p.scratch[rc.offset + row * rc.cols] = v;
                        if (!isfinite(v)) atomicOr(p.status, STATUS_NONFINITE);
                    });
            }
            __syncwarp();
        }
    }
    if (lane == 0) {
        p.Eout[g0] = E;
        p.Hout[g0] = H;
        p.Pout[g0] = P;
    }
    if (mine && i <= j) {
        p.Dout[(uint64_t) at * p.plane + g0] = xr;
        if (i < j) p.Dout[(uint64_t) (at + 1) * p.plane + g0] = xi;
    }
}

}  // namespace mbg
