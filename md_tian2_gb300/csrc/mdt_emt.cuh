// mdt_emt.cuh -- EMT energy/force for one bead inside a CTA (device code shared by
// the EMT kernels and the surrogate's EMT fallback).
#pragma once
#include "mdt_common.cuh"
#include "mdt_exp2tab.cuh"
#include "mdt_fastmath.cuh"

namespace mdt {

constexpr int kBlock = 128;  // threads per CTA (one trajectory per CTA)

// ---------------------------------------------------------------------------
// Arithmetic helpers.  On GB300 an FP64 instruction costs as much issue bandwidth as
// ~64 FP32 ones, so the FP64 kernels keep every FP64 operation that is not needed
// for 1e-10 eV/A parity off the FP64 pipe:
//  * reciprocal and reciprocal square root start from the hardware approximations
//    (rcp/rsqrt.approx.ftz.f64, good to ~2^-20) and are refined by one third-order step,
//    which cubes the relative error: accurate to ~1 ulp;
//  * conversions between FP64 and FP32 and FP64 comparisons run on the FP64 pipe too (measured
//    55 and 64 cycles per warp, an FP64 multiply-add 64, an integer instruction 1-2), so the
//    pair loops have none: floats are cut out of doubles by shifts (f32_of), ranges are tested
//    on high words, image shifts come from a table of their 27 vectors;
//  * the minimum-image shift (an integer per cell direction) is found in FP32 and
//    applied in FP64; when FP32 cannot decide the rounding (fractional part within
//    1e-4 of 1/2) the fractional coordinate is recomputed in FP64.
// ---------------------------------------------------------------------------
static __device__ __forceinline__ double rcp_nr(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);  // 1/x = y (1 + e + e^2 + ...)
    return fma(y, fma(e, e, e), y);
}

static __device__ __forceinline__ double rsqrt_nr(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y * y, 1.0);  // 1/sqrt(x) = y (1 + e/2 + 3 e^2/8 + ...)
    return fma(y * e, fma(e, 0.375, 0.5), y);
}

// n/d from the reciprocal id of d (within an ulp or two): the residual's correction makes the
// quotient round as a division does, in 3 FP64 instructions instead of about 10
static __device__ __forceinline__ double div_by(double n, double d, double id) {
    const double q = n * id;
    return fma(fma(-q, d, n), id, q);
}

// FP64 exp by the table-driven method of Tang (ACM TOMS 15(2), 1989): x = (512 n_hi + j)
// ln2/512 + r with |r| <= ln2/1024, exp(x) = 2^n_hi 2^(j/512) (1 + p(r)), p the Taylor series
// of exp(r) - 1 to r^4 (truncation below 2^-59).  ln2/512 enters in two parts (its double,
// then the remainder) so that r is exact to ~2^-100, and n = round(512 x / ln2) comes from
// adding 1.5 * 2^52.  10 FP64 instructions (13 with 64 entries and r^5, ~19 for exp()); the
// range test reads the high word, because a FP64 comparison costs as much as an addition.
// Outside [-700, 700], and for NaN, exp() itself.
static __device__ __forceinline__ double exp_t64(double x) {
    if ((__double2hiint(x) & 0x7fffffff) >= 0x4085e000) return exp(x);  // |x| >= 700
    const double shifter = 6755399441055744.0;
    const double t = fma(x, 738.65986093514926, shifter);
    const int n = __double2loint(t);
    const double nd = t - shifter;
    double r = fma(-nd, 0x1.62e42fefa39efp-10, x);
    r = fma(-nd, 0x1.abc9e3b39803fp-65, r);
    double q = fma(r, 1.0 / 24.0, 1.0 / 6.0);
    q = fma(r, q, 0.5);
    const double pr = fma(r * r, q, r);
    const double tj = __ldg(kExp2Tab + (n & 511));
    const double y = fma(tj, pr, tj);
    return __hiloint2double(__double2hiint(y) + (n >> 9) * (1 << 20), __double2loint(y));
}

template <typename R> struct Math;
template <> struct Math<double> {
    static __device__ __forceinline__ double ex(double x) { return exp_t64(x); }
    static __device__ __forceinline__ double rcp(double x) { return rcp_nr(x); }
    static __device__ __forceinline__ double rsq(double x) { return rsqrt_nr(x); }
};
template <> struct Math<float> {
    static __device__ __forceinline__ float ex(float x) { return __expf(x); }
    static __device__ __forceinline__ float rcp(float x) { return __frcp_rn(x); }
    static __device__ __forceinline__ float rsq(float x) { return rsqrtf(x); }
};

struct Cell;

template <typename R> struct SmemEmt {
    double *px, *py, *pz;  // staged bead positions
    float *xh, *yh, *zh, *xl, *yl, *zl;  // FP32 forces (R = float): their FP32 hi/lo split
    R *sig, *A, *fx, *fy, *fz;
    Cell *cell;
    int16_t *perm;         // atom of each staged place (places: species slot 0, slot 1, none)
    int *seg;              // first place of each of the three groups, N, runs per atom of slots 0 and 1
    double *red;           // 64 doubles for block reductions
    double *img;           // the 27 image-shift vectors of |n| <= 1 per direction (FP64 forces)
    double *cjk;           // the trajectory's normal-mode table, then its per-type, per-mode
                           // propagator tables (rp_cells doubles in all)
};

// doubles of the normal-mode area: the nb x nb table and 5 per-type, per-mode tables
__host__ __device__ constexpr size_t rp_cells(int max_beads) {
    return (size_t)max_beads * max_beads + 5 * (size_t)kMaxTypes * max_beads;
}

template <typename R>
static __device__ SmemEmt<R> carve_smem(unsigned char *base, int max_atoms, int max_beads) {
    SmemEmt<R> s;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        unsigned char *p = base + off;
        off += (bytes + 15) & ~size_t(15);
        return p;
    };
    s.px = (double *)take(sizeof(double) * max_atoms);
    s.py = (double *)take(sizeof(double) * max_atoms);
    s.pz = (double *)take(sizeof(double) * max_atoms);
    const size_t nf = sizeof(R) == 4 ? sizeof(float) * max_atoms : 0;
    s.xh = (float *)take(nf);
    s.yh = (float *)take(nf);
    s.zh = (float *)take(nf);
    s.xl = (float *)take(nf);
    s.yl = (float *)take(nf);
    s.zl = (float *)take(nf);
    s.red = (double *)take(sizeof(double) * 64);
    s.img = (double *)take(sizeof(double) * 81);
    s.cjk = (double *)take(sizeof(double) * rp_cells(max_beads));
    s.sig = (R *)take(sizeof(R) * max_atoms);
    s.A = (R *)take(sizeof(R) * max_atoms);
    s.fx = (R *)take(sizeof(R) * max_atoms);
    s.fy = (R *)take(sizeof(R) * max_atoms);
    s.fz = (R *)take(sizeof(R) * max_atoms);
    s.cell = (Cell *)take(256);
    s.perm = (int16_t *)take(sizeof(int16_t) * max_atoms);
    s.seg = (int *)take(sizeof(int) * 6);
    return s;
}

inline size_t smem_bytes(int max_atoms, int max_beads, size_t rsize) {
    auto r16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    return 3 * r16(8 * max_atoms) + (rsize == 4 ? 6 * r16(4 * max_atoms) : 0) + r16(8 * 64) + r16(8 * 81) +
           r16(8 * rp_cells(max_beads)) + 5 * r16(rsize * max_atoms) + 256 + r16(2 * max_atoms) + 32;
}

// Block-wide sum of a double; every thread gets the result.
static __device__ __noinline__ double block_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    double t = 0.0;
    for (int w = 0; w < nw; ++w) t += red[w];
    __syncthreads();
    return t;
}

// Block-wide sums of four doubles; every thread gets the results (red: 64 doubles, at most 16 warps).
static __device__ __noinline__ void block_sum4(double *v, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    for (int q = 0; q < 4; ++q)
        for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
    __syncthreads();
    if (lane == 0)
        for (int q = 0; q < 4; ++q) red[4 * warp + q] = v[q];
    __syncthreads();
    for (int q = 0; q < 4; ++q) {
        double t = 0.0;
        for (int w = 0; w < nw; ++w) t += red[4 * w + q];
        v[q] = t;
    }
    __syncthreads();
}

// Cell of one trajectory: FP64 matrix for applying image shifts, FP32 inverse for
// choosing them.  Column major (cell vectors as columns).
struct Cell {
    double h[9], hi[9];
    float hif[9], hf[9];  // FP32 inverse and (FP32 bead forces) FP32 matrix
    unsigned nz;  // bit k set when h[k] != 0
};
static_assert(sizeof(Cell) <= 256, "the shared-memory carve reserves 256 bytes for the cell");

// by the first warp of the CTA, nine lanes an entry each
static __device__ __forceinline__ void load_cell(const Batch &B, int t, Cell &c) {
    const int k = threadIdx.x;
    if (k >= 32) return;
    double h = 0.0;
    if (k < 9) {
        h = B.box[9 * (int64_t)t + k];
        const double hi = B.ibox[9 * (int64_t)t + k];
        c.h[k] = h;
        c.hi[k] = hi;
        c.hif[k] = (float)hi;
        c.hf[k] = (float)h;
    }
    const unsigned nz = __ballot_sync(0xffffffffu, h != 0.0);
    if (k == 0) c.nz = nz;
    __syncwarp();
}

// image index n = anint(w) for one fractional coordinate (Fortran anint: half away
// from zero).  FP32 decides unless it is within 1e-4 of a tie; then the fractional
// coordinate is recomputed in FP64 with the oracle's operation order and no fused
// multiply-add, so that exact ties (pairs half a cell apart on a perfect lattice) pick
// the same image on both sides.
static __device__ __forceinline__ double image_shift(float wf, const double *hi_row3, double ex, double ey, double ez,
                                                     int row) {
    const float n = roundf(wf);
    if (fabsf(fabsf(wf - n) - 0.5f) > 1e-4f) return (double)n;
    const double w = __dadd_rn(__dadd_rn(__dmul_rn(hi_row3[row], ex), __dmul_rn(hi_row3[row + 3], ey)),
                               __dmul_rn(hi_row3[row + 6], ez));
    return round(w);
}

// FP32 bead forces: the minimum image of r_i - r_j from the FP32 hi/lo split of the
// positions, with the image chosen as min_image chooses it (FP32, exact ties in FP64)
// and applied in FP32: no FP64 instruction per pair unless a pair sits on a tie.
template <typename S_>
static __device__ __forceinline__ void min_image_f(const Cell &c, const S_ &S, int i, int j, float &dx, float &dy,
                                            float &dz) {
    const float ex = (S.xh[i] - S.xh[j]) + (S.xl[i] - S.xl[j]);
    const float ey = (S.yh[i] - S.yh[j]) + (S.yl[i] - S.yl[j]);
    const float ez = (S.zh[i] - S.zh[j]) + (S.zl[i] - S.zl[j]);
    float n[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float w = c.hif[r] * ex + c.hif[r + 3] * ey + c.hif[r + 6] * ez;
        n[r] = roundf(w);
        if (!(fabsf(fabsf(w - n[r]) - 0.5f) > 1e-4f))
            n[r] = (float)image_shift(w, c.hi, S.px[i] - S.px[j], S.py[i] - S.py[j], S.pz[i] - S.pz[j], r);
    }
    dx = ex - (c.hf[0] * n[0] + c.hf[3] * n[1] + c.hf[6] * n[2]);
    dy = ey - (c.hf[1] * n[0] + c.hf[4] * n[1] + c.hf[7] * n[2]);
    dz = ez - (c.hf[2] * n[0] + c.hf[5] * n[1] + c.hf[8] * n[2]);
}

// minimum image of e = r_i - r_j, src/universe_mod.f90:411-428
static __device__ __forceinline__ void min_image(const Cell &c, double ex, double ey, double ez, double &dx, double &dy,
                                          double &dz) {
    const float fx = (float)ex, fy = (float)ey, fz = (float)ez;
    const float w0 = c.hif[0] * fx + c.hif[3] * fy + c.hif[6] * fz;
    const float w1 = c.hif[1] * fx + c.hif[4] * fy + c.hif[7] * fz;
    const float w2 = c.hif[2] * fx + c.hif[5] * fy + c.hif[8] * fz;
    const double n0 = image_shift(w0, c.hi, ex, ey, ez, 0);
    const double n1 = image_shift(w1, c.hi, ex, ey, ez, 1);
    const double n2 = image_shift(w2, c.hi, ex, ey, ez, 2);
    dx = ex;
    dy = ey;
    dz = ez;
    if (n0 != 0.0) {
        if (c.nz & 1u) dx = fma(-c.h[0], n0, dx);
        if (c.nz & 2u) dy = fma(-c.h[1], n0, dy);
        if (c.nz & 4u) dz = fma(-c.h[2], n0, dz);
    }
    if (n1 != 0.0) {
        if (c.nz & 8u) dx = fma(-c.h[3], n1, dx);
        if (c.nz & 16u) dy = fma(-c.h[4], n1, dy);
        if (c.nz & 32u) dz = fma(-c.h[5], n1, dz);
    }
    if (n2 != 0.0) {
        if (c.nz & 64u) dx = fma(-c.h[6], n2, dx);
        if (c.nz & 128u) dy = fma(-c.h[7], n2, dy);
        if (c.nz & 256u) dz = fma(-c.h[8], n2, dz);
    }
}

// the 27 shifts h n of |n| <= 1 per direction, entry 9 (n0 + 1) + 3 (n1 + 1) + (n2 + 1); by the
// first warp, after load_cell
static __device__ __forceinline__ void image_table(const Cell &c, double *img) {
    const int k = threadIdx.x;
    if (k >= 27) return;
    const double n0 = k / 9 - 1, n1 = k / 3 % 3 - 1, n2 = k % 3 - 1;
    for (int d = 0; d < 3; ++d) img[3 * k + d] = fma(c.h[d], n0, fma(c.h[d + 3], n1, c.h[d + 6] * n2));
}

// min_image with its shift from the table: no FP64 conversion, comparison or product.  A
// fractional coordinate near a tie, or an image further away, takes min_image itself.
static __device__ __forceinline__ void min_image_t(const Cell &c, const double *img, double ex, double ey, double ez,
                                                   double &dx, double &dy, double &dz) {
    const float fx = f32_of(ex), fy = f32_of(ey), fz = f32_of(ez);
    int n[3];
    bool plain = true;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float w = c.hif[r] * fx + c.hif[r + 3] * fy + c.hif[r + 6] * fz;
        const float f = rintf(w);
        plain = plain && fabsf(fabsf(w - f) - 0.5f) > 1e-4f && fabsf(f) <= 1.f;
        n[r] = (int)f;
    }
    dx = ex;
    dy = ey;
    dz = ez;
    if (plain) {
        const int k = 9 * n[0] + 3 * n[1] + n[2] + 13;
        if (k != 13) {
            dx -= img[3 * k];
            dy -= img[3 * k + 1];
            dz -= img[3 * k + 2];
        }
    } else {
        min_image(c, ex, ey, ez, dx, dy, dz);
    }
}

// ---------------------------------------------------------------------------
// EMT for one bead of one trajectory.  Adds forces into B.f* (stores them when `store`), sets
// dens, adds the bead's energy into B.epot.  Must be called by all threads of the CTA.
//
// Atoms are staged by species: places [seg[0], seg[1]) hold the atoms of species slot 0,
// [seg[1], seg[2]) those of slot 1, the rest are not EMT.  Almost every pair has two atoms of
// the metal, so pairs are walked per species with the species' constants in registers and no
// branch; the few pairs of the two species run in a loop of their own (in one common walk nearly
// every warp met one of them, and took both branches).
//
// Pairs of one species (M atoms): (i, j = (i+k) mod M), k = 1..M/2, in scratch slot
// (k-1) M + i (the k = M/2 row holds only i < M/2 when M is even).  A thread takes one atom i
// and a run of k: its side of a pair sums in registers, the other side is read back from the
// scratch by the thread that owns j (lanes hold consecutive i: every access coalesces).  A
// shared-memory FP64 addition costs 137 cycles a warp, reading the value back 5.
//   pass 1  distance, density term rho, pair energy, and the scalars q = -rho'/r, fv of the force
//   epilogue (per atom) sigma -> s, cohesive energy, embedded density, A = (dE/ds)/(beta eta2 sigma)
//   pass 2  cc = (A_i + A_j) q + fv, force += cc d on i; cc left in q's slot; then -cc d on j
// ---------------------------------------------------------------------------
template <typename R> struct PairK {
    R acut, rcut, eta, etaq, b, kb, g, c;
};

// cutoff function theta and acut e theta (its logarithmic derivative) at distance r
template <typename R> static __device__ __forceinline__ void emt_theta(R acut, R rcut, R r, R &theta, R &rt1) {
    const R x = acut * (r - rcut);
    if constexpr (sizeof(R) == 8) {
        // x < -41: 1 + e rounds to 1 and acut e is below half an ulp of eta and kappa/beta
        const unsigned h = (unsigned)__double2hiint(x);
        if (h > 0xc0448000u && h < 0xfff00000u) {
            theta = 1.0;
            rt1 = 0.0;
            return;
        }
    }
    const R e = Math<R>::ex(x);
    theta = Math<R>::rcp(R(1) + e);
    rt1 = acut * e * theta;
}

// running sum of pair energies: FP64, or an FP32 sum with its rounding errors kept beside it
// (48 bits; an FP64 addition of a float costs two FP64-pipe slots a pair)
template <typename R> struct EnergySum;
template <> struct EnergySum<double> {
    double s = 0.0;
    __device__ __forceinline__ void add(double x) { s += x; }
    __device__ __forceinline__ double value() const { return s; }
};
template <> struct EnergySum<float> {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
        c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z)));
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

__device__ __forceinline__ bool is_zero(double x) {
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }

// displacement (minimum image) of staged places i, j
template <typename R>
static __device__ __forceinline__ void place_diff(const SmemEmt<R> &S, int i, int j, R &rx, R &ry, R &rz) {
    if constexpr (sizeof(R) == 4)
        min_image_f(*S.cell, S, i, j, rx, ry, rz);
    else
        min_image_t(*S.cell, S.img, S.px[i] - S.px[j], S.py[i] - S.py[j], S.pz[i] - S.pz[j], rx, ry, rz);
}

// Beyond the cutoff, like the reference's `if (r > cutoff*rcut) cycle` (pes_emt_mod.f90:660): a
// distance that is not a number enters the sums.  FP64: on the high words, the exact comparison
// only when they are equal.
static __device__ __forceinline__ bool beyond(double r2, double cut2) {
    const int a = __double2hiint(r2), c = __double2hiint(cut2);
    return a == c ? r2 > cut2 : a > c && a <= 0x7ff00000;
}
static __device__ __forceinline__ bool beyond(float r2, float cut2) { return r2 > cut2; }

// Runs of k per atom (1..16) so that the M C work items of the pair loops fill the CTA's rounds
// best (cost: rounds x run length; a run also pays its sums once).  One warp, lane = candidate.
static __device__ __forceinline__ int pair_chunks(int M, int nt) {
    const int C = (threadIdx.x & 15) + 1, K = M / 2;
    const int cost = C <= K || C == 1 ? ((M * C + nt - 1) / nt) * (2 * ((K + C - 1) / C) + 1) : 1 << 26;
    const int best = __reduce_min_sync(0xffffffffu, cost << 4 | (C - 1));
    return (best & 15) + 1;
}

template <typename R>
static __device__ void emt_bead(const Batch &B, const EmtConst &E, const SmemEmt<R> &S, int t, int b,
                         bool do_forces, bool store = false) {
    const int N = B.natoms[t];
    const int64_t base = B.ba_off[t] + (int64_t)b * N;
    const int aoff = B.atom_off[t];
    const int tid = threadIdx.x, nt = blockDim.x;

    // ---- staging: places by species (identity when the atoms come sorted, as
    // merge_universes makes them: projectile first) ------------------------------------
    auto group = [&](int i) {
        const int s = E.slot_of_type[B.type[aoff + i]];
        return s < 0 ? 2 : s;
    };
    bool unsorted = false;
    for (int i = tid; i < N; i += nt) {
        const int g = group(i), h = i ? group(i - 1) : -1;
        unsorted |= h > g;
        for (int k = h + 1; k <= g; ++k) S.seg[k] = i;
        if (i == N - 1)
            for (int k = g + 1; k <= 3; ++k) S.seg[k] = N;
        S.perm[i] = (int16_t)i;
    }
    load_cell(B, t, *S.cell);
    if constexpr (sizeof(R) == 8) image_table(*S.cell, S.img);
    if (__syncthreads_or(unsorted)) {
        if (tid == 0) {
            int p = 0;
            for (int g = 0; g < 3; ++g) {
                S.seg[g] = p;
                for (int i = 0; i < N; ++i)
                    if (group(i) == g) S.perm[p++] = (int16_t)i;
            }
            S.seg[3] = N;
        }
        __syncthreads();
    }
    for (int p = tid; p < N; p += nt) {
        const int64_t k = base + S.perm[p];
        const double x = B.rx[k], y = B.ry[k], z = B.rz[k];
        S.px[p] = x;
        S.py[p] = y;
        S.pz[p] = z;
        if constexpr (sizeof(R) == 4) {
            S.xh[p] = (float)x;
            S.yh[p] = (float)y;
            S.zh[p] = (float)z;
            S.xl[p] = (float)(x - (double)S.xh[p]);
            S.yl[p] = (float)(y - (double)S.yh[p]);
            S.zl[p] = (float)(z - (double)S.zh[p]);
        }
        S.sig[p] = R(0);
        S.A[p] = R(0);
        S.fx[p] = R(0);
        S.fy[p] = R(0);
        S.fz[p] = R(0);
    }
    if (tid < 32) {
        const int c0 = pair_chunks(S.seg[1], nt), c1 = pair_chunks(S.seg[2] - S.seg[1], nt);
        if (tid == 0) {
            S.seg[4] = c0;
            S.seg[5] = c1;
        }
    }
    __syncthreads();
    const int n0 = S.seg[1], n1 = S.seg[2] - S.seg[1];
    const int chunks[2] = {S.seg[4], S.seg[5]};

    const int NK = N * (N / 2);
    R *scr = (R *)B.pair_scratch + 6 * (B.pair_off[t] + (int64_t)b * NK);
    R *s_dx = scr, *s_dy = scr + NK, *s_dz = scr + 2 * NK, *s_q = scr + 3 * NK, *s_fv = scr + 4 * NK,
      *s_rho = scr + 5 * NK;
    const R cut2 = (R)E.cut2;
    EnergySum<R> e_pair;

    // ---- pass 1, pairs of one species -------------------------------------------------
    for (int s = 0, off = 0; s < E.nspecies; ++s) {
        const int m0 = S.seg[s], M = S.seg[s + 1] - m0, K = M / 2;
        if (K == 0) continue;
        // QUIRK kept from pes_emt_mod.f90:705: the type1-type1 density derivative uses eta2 of
        // type2.
        const PairK<R> k{(R)E.acut,    (R)E.rcut,          (R)E.eta2[s],    (R)E.eta2[E.hh_quirk && s == 0 ? 1 : s],
                         (R)E.betas0[s], (R)E.kappadbeta[s], (R)E.igamma1[s], (R)E.g2v0[s]};
        const int C = chunks[s], per = (K + C - 1) / C;
        for (int w = tid; w < M * C; w += nt) {
            const int c = w / M, i = w - c * M;
            const int k1 = min((c + 1) * per, (2 * K == M && i >= K) ? K - 1 : K);
            R acc = R(0);
            for (int kk = 1 + c * per; kk <= k1; ++kk) {
                int j = i + kk;
                if (j >= M) j -= M;
                const int p = off + (kk - 1) * M + i;
                R q = R(0), fv = R(0), rho = R(0), rx, ry, rz;
                place_diff<R>(S, m0 + i, m0 + j, rx, ry, rz);
                const R r2 = rx * rx + ry * ry + rz * rz;
                if (!beyond(r2, cut2)) {
                    const R ir = Math<R>::rsq(r2), r = r2 * ir;
                    R theta, rt1;
                    emt_theta<R>(k.acut, k.rcut, r, theta, rt1);
                    const R phi = theta * Math<R>::ex(-k.eta * (r - k.b));
                    const R psi = theta * Math<R>::ex(-k.kb * (r - k.b));
                    rho = k.g * phi;
                    acc += rho;
                    e_pair.add(-(k.c * psi));
                    q = k.g * (k.etaq + rt1) * phi * ir;
                    fv = -(k.c * (k.kb + rt1) * psi * ir);
                }
                s_rho[p] = rho;
                if (do_forces) {
                    s_dx[p] = rx;
                    s_dy[p] = ry;
                    s_dz[p] = rz;
                    s_q[p] = q;
                    s_fv[p] = fv;
                }
            }
            if (C == 1) S.sig[m0 + i] = acc;
            else atomicAdd(&S.sig[m0 + i], acc);
        }
        off += M * (M - 1) / 2;
    }
    // ---- pass 1, pairs of the two species: a warp's lanes over the slot-1 atoms ----------
    const int t0 = E.type_of_slot[0], t1 = E.type_of_slot[1];
    const int xoff = n0 * (n0 - 1) / 2 + n1 * (n1 - 1) / 2;  // cross pairs follow in the scratch
    __syncthreads();
    for (int a = 0; a < n0 && n1 > 0; ++a) {
        const int ia = S.perm[a];
        R sa = R(0);
        for (int jj = tid; jj < n1; jj += nt) {
            const int j = n0 + jj, p = xoff + a * n1 + jj;
            R q_a = R(0), q_j = R(0), fv = R(0), rx = R(0), ry = R(0), rz = R(0);
            // pes(ti, tj) of the pair's first atom in the (i, i+k mod N) order, should the table not
            // be symmetric
            const int d = S.perm[j] - ia, dk = d > 0 ? d : d + N;
            const bool a_first = 2 * dk < N || (2 * dk == N && ia < S.perm[j]);
            if ((E.pair_mask >> (a_first ? t0 * kMaxTypes + t1 : t1 * kMaxTypes + t0)) & 1u) {
                place_diff<R>(S, a, j, rx, ry, rz);
                const R r2 = rx * rx + ry * ry + rz * rz;
                if (!beyond(r2, cut2)) {
                    const R ir = Math<R>::rsq(r2), r = r2 * ir;
                    R theta, rt1;
                    emt_theta<R>((R)E.acut, (R)E.rcut, r, theta, rt1);
                    const R phi_j = theta * Math<R>::ex(-(R)E.eta2[1] * (r - (R)E.betas0[1]));
                    const R psi_j = theta * Math<R>::ex(-(R)E.kappadbeta[1] * (r - (R)E.betas0[1]));
                    const R phi_a = theta * Math<R>::ex(-(R)E.eta2[0] * (r - (R)E.betas0[0]));
                    const R psi_a = theta * Math<R>::ex(-(R)E.kappadbeta[0] * (r - (R)E.betas0[0]));
                    const R gaj = (R)(E.igamma1[0] * E.chi[0][1]), gja = (R)(E.igamma1[1] * E.chi[1][0]);
                    const R caj = (R)(E.g2v0[0] * E.chi[0][1]), cja = (R)(E.g2v0[1] * E.chi[1][0]);
                    sa += gaj * phi_j;
                    S.sig[j] += gja * phi_a;  // this thread alone owns j here
                    e_pair.add(-R(0.5) * (caj * psi_j + cja * psi_a));
                    fv = -R(0.5) * (caj * ((R)E.kappadbeta[1] + rt1) * psi_j +
                                    cja * ((R)E.kappadbeta[0] + rt1) * psi_a) * ir;
                    q_a = gaj * ((R)E.eta2[1] + rt1) * phi_j * ir;
                    q_j = gja * ((R)E.eta2[0] + rt1) * phi_a * ir;
                }
            }
            if (do_forces) {
                s_dx[p] = rx;
                s_dy[p] = ry;
                s_dz[p] = rz;
                s_q[p] = q_a;
                s_fv[p] = fv;
                s_rho[p] = q_j;
            }
        }
        for (int o = 16; o > 0; o >>= 1) sa += __shfl_xor_sync(0xffffffffu, sa, o);
        if ((tid & 31) == 0 && !is_zero(sa)) atomicAdd(&S.sig[a], sa);
    }
    __syncthreads();
    // ---- densities, the other side of each pair ----------------------------------------
    for (int s = 0, off = 0; s < E.nspecies; ++s) {
        const int m0 = S.seg[s], M = S.seg[s + 1] - m0, K = M / 2;
        if (K == 0) continue;
        const int C = chunks[s], per = (K + C - 1) / C;
        for (int w = tid; w < M * C; w += nt) {
            const int c = w / M, j = w - c * M;
            const int k1 = min((c + 1) * per, K);
            R acc = R(0);
            for (int kk = 1 + c * per; kk <= k1; ++kk) {
                int m = j - kk;
                if (m < 0) m += M;
                if (2 * kk == M && m >= K) continue;
                const R rho = s_rho[off + (kk - 1) * M + m];
                if (!is_zero(rho)) acc += rho;
            }
            atomicAdd(&S.sig[m0 + j], acc);
        }
        off += M * (M - 1) / 2;
    }
    __syncthreads();

    // ---- per-atom epilogue ---------------------------------------------------
    double e_atom = 0.0;
    for (int i = tid; i < n0 + n1; i += nt) {
        const int s = i >= n0;
        double sc = (double)S.sig[i], cl = sc;
        // above 1e-9 (by its high word) neither floor of pes_emt_mod.f90:793 acts
        if (__double2hiint(sc) <= 0x3e112e0b || __double2hiint(sc) >= 0x7ff00000) {
            sc = fmax((double)1e-30f, sc);  // single-precision 1e-30
            cl = fmax(kTolerance, sc);
        }
        const double be = E.betaeta2[s], sa = div_by(-log(cl * kTwelfth), be, E.ibe[s]);
        const double lsa = E.lambda[s] * sa, el = exp_t64(-lsa), ek = exp_t64(-E.kappa[s] * sa);
        e_atom += E.e0[s] * (fma(lsa, el, el) - 1.0) + E.v6[s] * ek;
        const double bs = be * sc;
        S.A[i] = (R)div_by(E.e0l2[s] * sa * el + E.v6k[s] * ek, bs, rcp_nr(bs));
        B.dens[base + S.perm[i]] = E.n0[s] * exp_t64(E.dens_exp[s] * sa);
    }
    const double etot = block_sum(e_pair.value() + e_atom, S.red);  // contains __syncthreads
    if (tid == 0) B.epot[B.bead_off[t] + b] += etot;
    if (!do_forces) return;

    // ---- pass 2 ----------------------------------------------------------------------
    for (int s = 0, off = 0; s < E.nspecies; ++s) {  // the first atom's side
        const int m0 = S.seg[s], M = S.seg[s + 1] - m0, K = M / 2;
        if (K == 0) continue;
        const int C = chunks[s], per = (K + C - 1) / C;
        for (int w = tid; w < M * C; w += nt) {
            const int c = w / M, i = w - c * M;
            const int k1 = min((c + 1) * per, (2 * K == M && i >= K) ? K - 1 : K);
            const R Ai = S.A[m0 + i];
            R fx = R(0), fy = R(0), fz = R(0);
            for (int kk = 1 + c * per; kk <= k1; ++kk) {
                int j = i + kk;
                if (j >= M) j -= M;
                const int p = off + (kk - 1) * M + i;
                const R q = s_q[p], fv = s_fv[p];
                if (is_zero(q) && is_zero(fv)) continue;  // beyond the cutoff: q's slot holds the 0
                const R cc = Ai * q + S.A[m0 + j] * q + fv;
                s_q[p] = cc;
                fx += cc * s_dx[p];
                fy += cc * s_dy[p];
                fz += cc * s_dz[p];
            }
            if (C == 1) {
                S.fx[m0 + i] = fx;
                S.fy[m0 + i] = fy;
                S.fz[m0 + i] = fz;
            } else {
                atomicAdd(&S.fx[m0 + i], fx);
                atomicAdd(&S.fy[m0 + i], fy);
                atomicAdd(&S.fz[m0 + i], fz);
            }
        }
        off += M * (M - 1) / 2;
    }
    __syncthreads();
    for (int a = 0; a < n0 && n1 > 0; ++a) {  // pairs of the two species
        const R Aa = S.A[a];
        R fx = R(0), fy = R(0), fz = R(0);
        for (int jj = tid; jj < n1; jj += nt) {
            const int j = n0 + jj, p = xoff + a * n1 + jj;
            const R cc = Aa * s_q[p] + S.A[j] * s_rho[p] + s_fv[p];
            const R gx = cc * s_dx[p], gy = cc * s_dy[p], gz = cc * s_dz[p];
            fx += gx;
            fy += gy;
            fz += gz;
            S.fx[j] -= gx;  // this thread alone owns j here
            S.fy[j] -= gy;
            S.fz[j] -= gz;
        }
        for (int o = 16; o > 0; o >>= 1) {
            fx += __shfl_xor_sync(0xffffffffu, fx, o);
            fy += __shfl_xor_sync(0xffffffffu, fy, o);
            fz += __shfl_xor_sync(0xffffffffu, fz, o);
        }
        if ((tid & 31) == 0) {
            atomicAdd(&S.fx[a], fx);
            atomicAdd(&S.fy[a], fy);
            atomicAdd(&S.fz[a], fz);
        }
    }
    __syncthreads();
    for (int s = 0, off = 0; s < E.nspecies; ++s) {  // the second atom's side
        const int m0 = S.seg[s], M = S.seg[s + 1] - m0, K = M / 2;
        if (K == 0) continue;
        const int C = chunks[s], per = (K + C - 1) / C;
        for (int w = tid; w < M * C; w += nt) {
            const int c = w / M, j = w - c * M;
            const int k1 = min((c + 1) * per, K);
            R fx = R(0), fy = R(0), fz = R(0);
            for (int kk = 1 + c * per; kk <= k1; ++kk) {
                int m = j - kk;
                if (m < 0) m += M;
                if (2 * kk == M && m >= K) continue;
                const int p = off + (kk - 1) * M + m;
                const R cc = s_q[p];
                if (is_zero(cc)) continue;
                fx -= cc * s_dx[p];
                fy -= cc * s_dy[p];
                fz -= cc * s_dz[p];
            }
            atomicAdd(&S.fx[m0 + j], fx);
            atomicAdd(&S.fy[m0 + j], fy);
            atomicAdd(&S.fz[m0 + j], fz);
        }
        off += M * (M - 1) / 2;
    }
    __syncthreads();
    for (int p = tid; p < N; p += nt) {
        const int64_t k = base + S.perm[p];
        if (store) {
            B.fx[k] = (double)S.fx[p];
            B.fy[k] = (double)S.fy[p];
            B.fz[k] = (double)S.fz[p];
        } else {
            B.fx[k] += (double)S.fx[p];
            B.fy[k] += (double)S.fy[p];
            B.fz[k] += (double)S.fz[p];
        }
    }
    __syncthreads();
}

}  // namespace mdt
