// mdt_emt.cuh -- EMT energy/force for one bead inside a CTA (device code shared by
// the EMT kernels and the surrogate's EMT fallback).
#pragma once
#include "mdt_common.cuh"
#include "mdt_fastmath.cuh"

namespace mdt {

constexpr int kBlock = 128;      // threads per CTA (one trajectory per CTA)
constexpr int kWideBlock = 256;  // the same for batches of at most one trajectory per SM

// ---------------------------------------------------------------------------
// Arithmetic helpers.  On GB300 an FP64 instruction costs as much issue bandwidth as
// ~64 FP32 ones, so the FP64 kernels keep every FP64 operation that is not needed
// for 1e-10 eV/A parity off the FP64 pipe:
//  * reciprocal and reciprocal square root start from the hardware approximations
//    (rcp/rsqrt.approx.ftz.f64, good to ~2^-20) and are refined by one third-order step,
//    which cubes the relative error: accurate to ~1 ulp;
//  * conversions between FP64 and FP32 and FP64 comparisons run on the FP64 pipe too (measured
//    55 and 64 cycles per warp, an FP64 multiply-add 64, an integer instruction 1-2), so the
//    pair loops have none: floats are cut out of doubles by shifts (f32_screen), ranges are tested
//    on high words, image shifts come from a table of their 27 vectors;
//  * the minimum-image shift (an integer per cell direction) is found in FP32 and
//    applied in FP64; when FP32 cannot decide the rounding (fractional part within
//    1e-4 of 1/2) the fractional coordinate is recomputed in FP64.
// ---------------------------------------------------------------------------
template <typename R> struct Math;
template <> struct Math<double> {
    static __device__ __forceinline__ double ex(double x) { return exp_t64(x); }
    static __device__ __forceinline__ double rcp(double x) { return rcp_nr(x); }
    static __device__ __forceinline__ double rsq(double x) { return rsqrt_nr(x); }
};
// FP32: the hardware approximations behind __expf and rsqrtf without their steps for denormal
// operands (results below 2^-126 flush to zero).  The reciprocal stays the correctly rounded one:
// embedding and pair forces cancel to a hundredth, and a reciprocal one bit off in some pairs moved
// the forces of the FP32 ring-polymer batch by 2.3e-5 instead of 1.2e-5 (relative; their FP32 error
// is 1.8e-5).
template <> struct Math<float> {
    static __device__ __forceinline__ float ex(float x) { return ex2a(x * kLog2eF); }
    static __device__ __forceinline__ float rcp(float x) { return __frcp_rn(x); }
    static __device__ __forceinline__ float rsq(float x) {
        float y;
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    }
};

struct Cell;

template <typename R> struct SmemEmt {
    double *px, *py, *pz;  // staged bead positions
    float4 *ph, *pl;       // FP32 forces (R = float): their FP32 hi/lo split
    R *sig, *A, *fx, *fy, *fz;
    Cell *cell;
    double *en;            // per place: the bead's energies (several beads at a time; else null)
    int places;            // staged atoms the arrays hold (beads at a time x atoms)
    size_t bytes;          // all of it
    int16_t *perm;         // atom of each place of a bead (places: species slot 0, slot 1, none)
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

// Sizes of the EMT code's shared memory: what carve_smem lays out and smem_bytes adds up.
struct EmtLayout {
    int max_atoms, max_beads;
    int places;     // staged atoms
    bool together;  // beads several at a time: an energy per place
    bool img;       // the image-shift table
};

// The EMT kernels evaluate the beads of a ring polymer several at a time (their per-atom FP64 work
// fills warps, and the CTA's barriers are shared), up to 512 staged atoms: as many as fit, which is
// more for the small trajectories of a batch than for its largest (emt_group).  Above 512 atoms one
// at a time, and without the image table: there the positions and sums may reach the shared-memory limit.
__host__ __device__ constexpr EmtLayout emt_layout(int max_atoms, int max_beads) {
    return EmtLayout{max_atoms, max_beads,
                     max_atoms * max_beads <= 512 ? max_atoms * max_beads
                     : max_atoms <= 512           ? 512 / max_atoms * max_atoms
                                                  : max_atoms,
                     max_beads > 1 && max_atoms <= 512, max_atoms <= 512};
}

// One bead at a time, without the image table: the network kernels' fallback, whose shared memory bounds the
// models and sizes that fit, and the allocation-free call.
__host__ __device__ constexpr EmtLayout emt_layout_one(int max_atoms, int max_beads) {
    return EmtLayout{max_atoms, max_beads, max_atoms, false, false};
}

// Work of a batch with teams of 1, 2, 4, 8 CTAs per trajectory, in pairs of atoms: CTA time it takes up
// (a CTA of a team waits where the trajectory has fewer beads) and its longest trajectory's.
struct TeamWork {
    double all[4], longest[4];
    void add(int natoms, int nbeads) {
        for (int k = 0; k < 4; ++k) {
            const int rounds = (nbeads + (1 << k) - 1) >> k;
            const double w = (double)rounds * natoms * natoms;
            all[k] += w * (1 << k);
            longest[k] = longest[k] > w ? longest[k] : w;
        }
    }
};

// CTAs per trajectory of a ring-polymer batch (log2), `slots` of them resident: doubled while it brings the batch's
// end nearer (its longest trajectory and an even share of all work), has beads to share and leaves at most
// four waves.  With one CTA per trajectory a batch waits for its longest ring polymer (32 beads, one after the
// other): 96 FP64 trajectories 31.3 ms with one, 13.1 with 8; 1024 with FP32 forces 26.3 ms with one, 22.4
// with 2, 33 with 4 (fewer beads at a time fill fewer warps, and every CTA repeats the tables and sums of a
// step).  1199 single beads beside one 2-bead ring polymer, five FP64 steps: 1.2 ms with one, 2.5 with 2 (half the
// CTAs wait).
inline int team_log2(const TeamWork &w, int64_t ntraj, int max_beads, int64_t slots) {
    int k = 0;
    while (k < 3 && (2 << k) <= max_beads && ntraj * (2 << k) <= 4 * slots &&
           w.longest[k + 1] + w.all[k + 1] / slots < w.longest[k] + w.all[k] / slots)
        ++k;
    return k;
}

// beads of an N-atom trajectory evaluated together, at most `per`
__host__ __device__ constexpr int emt_group(int places, bool together, int N, int per) {
    return !together ? 1 : per < places / N ? per : places / N;
}

template <typename R>
static __host__ __device__ SmemEmt<R> carve_smem(unsigned char *base, const EmtLayout &L) {
    SmemEmt<R> s;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        unsigned char *p = base + off;
        off += (bytes + 15) & ~size_t(15);
        return p;
    };
    const int places = L.places;
    const int dp = sizeof(R) == 8 ? places : 0;  // FP64 forces: FP64 positions; FP32: their hi/lo split
    s.places = places;
    s.px = (double *)take(sizeof(double) * dp);
    s.py = (double *)take(sizeof(double) * dp);
    s.pz = (double *)take(sizeof(double) * dp);
    const size_t nf = sizeof(R) == 4 ? sizeof(float4) * places : 0;
    s.ph = (float4 *)take(nf);
    s.pl = (float4 *)take(nf);
    s.red = (double *)take(sizeof(double) * 64);
    s.img = (double *)take(L.img ? sizeof(double) * 81 : 0);
    if (!L.img) s.img = nullptr;
    s.cjk = (double *)take(sizeof(double) * rp_cells(L.max_beads));
    s.sig = (R *)take(sizeof(R) * places);
    s.A = (R *)take(sizeof(R) * places);
    s.fx = (R *)take(sizeof(R) * places);
    s.fy = (R *)take(sizeof(R) * places);
    s.fz = (R *)take(sizeof(R) * places);
    s.en = (double *)take(L.together ? sizeof(double) * places : 0);
    if (!L.together) s.en = nullptr;
    unsigned char *const cell = take(256);
    s.cell = (Cell *)cell;
    s.seg = (int *)(cell + 224);
    s.perm = (int16_t *)take(sizeof(int16_t) * L.max_atoms);
    s.bytes = off;
    return s;
}

// (the layout from an address of no meaning, for its size)
template <typename R> inline size_t smem_bytes(const EmtLayout &L) {
    return carve_smem<R>(reinterpret_cast<unsigned char *>(uintptr_t(256)), L).bytes;
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
static_assert(sizeof(Cell) <= 224, "the shared-memory carve reserves 224 bytes for the cell, 32 for the groups");

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

// all three image indices of a pair of which one sits on a tie
static __device__ __noinline__ float3 image_exact(const Cell &c, float3 w, double ex, double ey, double ez) {
    return make_float3((float)image_shift(w.x, c.hi, ex, ey, ez, 0), (float)image_shift(w.y, c.hi, ex, ey, ez, 1),
                       (float)image_shift(w.z, c.hi, ex, ey, ez, 2));
}

// nearest integer of an image coordinate |w| < 2^21 (ties to even; the caller treats ties)
static __device__ __forceinline__ float image_round(float w) { return (w + 12582912.f) - 12582912.f; }

// Minimum image of one staged place against others, the place and the cell held in registers (the
// pair loops write the scratch, so nothing read through pointers stays in a register by itself).
template <typename R> struct PlaceDiff;

// FP32 forces, from the FP32 hi/lo split of the positions, with the image chosen as min_image
// chooses it (FP32, exact ties in FP64) and applied in FP32: no FP64 instruction per pair unless
// a pair sits on a tie.
template <> struct PlaceDiff<float> {
    float xh, yh, zh, xl, yl, zl, h[9], hi[9];
    int i;
    bool slab;                   // in-plane cell vectors and one along z: the other entries are zero
    const double *rx, *ry, *rz;  // positions of the bead in global memory (ties)
    const int16_t *perm;
    const Cell *cell;
    template <typename S_>
    __device__ __forceinline__ PlaceDiff(const Batch &B, const S_ &S, int64_t base0)
        : rx(B.rx + base0), ry(B.ry + base0), rz(B.rz + base0), perm(S.perm), cell(S.cell) {
#pragma unroll
        for (int k = 0; k < 9; ++k) {
            h[k] = S.cell->hf[k];
            hi[k] = S.cell->hif[k];
        }
        slab = h[2] == 0.f && h[5] == 0.f && h[6] == 0.f && h[7] == 0.f && hi[2] == 0.f && hi[5] == 0.f &&
               hi[6] == 0.f && hi[7] == 0.f;
    }
    template <typename S_> __device__ __forceinline__ void set(const S_ &S, int place) {
        i = place;
        const float4 a = S.ph[place], b = S.pl[place];
        xh = a.x;
        yh = a.y;
        zh = a.z;
        xl = b.x;
        yl = b.y;
        zl = b.z;
    }
    // N: atoms of a bead; places i and j belong to the same one
    template <typename S_>
    __device__ __forceinline__ void diff(const S_ &S, int j, int N, float &dx, float &dy, float &dz) const {
        const float4 a = S.ph[j], b = S.pl[j];
        const float ex = (xh - a.x) + (xl - b.x), ey = (yh - a.y) + (yl - b.y), ez = (zh - a.z) + (zl - b.z);
        float n[3], w[3];
        if (slab) {  // the same sums without their zero terms
            w[0] = hi[0] * ex + hi[3] * ey;
            w[1] = hi[1] * ex + hi[4] * ey;
            w[2] = hi[8] * ez;
        } else {
#pragma unroll
            for (int r = 0; r < 3; ++r) w[r] = hi[r] * ex + hi[r + 3] * ey + hi[r + 6] * ez;
        }
#pragma unroll
        for (int r = 0; r < 3; ++r) n[r] = image_round(w[r]);
        const float off = fmaxf(fabsf(w[0] - n[0]), fmaxf(fabsf(w[1] - n[1]), fabsf(w[2] - n[2])));
        const float big = fmaxf(fabsf(w[0]), fmaxf(fabsf(w[1]), fabsf(w[2])));
        if (!(off < 0.4999f && big < 2097152.f)) {
            const int g = i / N * N;  // the bead's slots follow each other as its places do
            const int64_t p = g + perm[i - g], q = g + perm[j - g];
            const float3 m = image_exact(*cell, make_float3(w[0], w[1], w[2]), rx[p] - rx[q], ry[p] - ry[q], rz[p] - rz[q]);
            n[0] = m.x;
            n[1] = m.y;
            n[2] = m.z;
        }
        if (slab) {
            dx = ex - (h[0] * n[0] + h[3] * n[1]);
            dy = ey - (h[1] * n[0] + h[4] * n[1]);
            dz = ez - h[8] * n[2];
        } else {
            dx = ex - (h[0] * n[0] + h[3] * n[1] + h[6] * n[2]);
            dy = ey - (h[1] * n[0] + h[4] * n[1] + h[7] * n[2]);
            dz = ez - (h[2] * n[0] + h[5] * n[1] + h[8] * n[2]);
        }
    }
};

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

static __device__ __noinline__ double3 min_image_far(const Cell &c, double ex, double ey, double ez) {
    double3 d;
    min_image(c, ex, ey, ez, d.x, d.y, d.z);
    return d;
}

// the 27 shifts h n of |n| <= 1 per direction, entry 9 (n0 + 1) + 3 (n1 + 1) + (n2 + 1); by the
// first warp, after load_cell
static __device__ __forceinline__ void image_table(const Cell &c, double *img) {
    const int k = threadIdx.x;
    if (k >= 27 || !img) return;
    const double n0 = k / 9 - 1, n1 = k / 3 % 3 - 1, n2 = k % 3 - 1;
    for (int d = 0; d < 3; ++d) img[3 * k + d] = fma(c.h[d], n0, fma(c.h[d + 3], n1, c.h[d + 6] * n2));
}

// e minus the shift of |n| <= 1 per direction, without the table (large trajectories, the network
// kernels' fallback)
static __device__ __noinline__ double3 image_near(const Cell &c, float n0, float n1, float n2, double ex, double ey,
                                                  double ez) {
    const float n[3] = {n0, n1, n2};
    double d[3] = {ex, ey, ez};
#pragma unroll
    for (int v = 0; v < 3; ++v) {
        if (n[v] == 0.f) continue;
        const double m = n[v] < 0.f ? 1.0 : -1.0;
#pragma unroll
        for (int q = 0; q < 3; ++q)
            if (c.nz >> (3 * v + q) & 1u) d[q] = fma(c.h[3 * v + q], m, d[q]);
    }
    return make_double3(d[0], d[1], d[2]);
}

// FP64 forces: min_image with its shift from the table: no FP64 conversion, comparison or product, and
// nothing at all for a pair whose nearest image is its own.
// A fractional coordinate near a tie, or an image further away, takes min_image itself.
template <> struct PlaceDiff<double> {
    double x, y, z;
    float hi[9];
    const Cell *cell;
    const double *img;
    template <typename S_>
    __device__ __forceinline__ PlaceDiff(const Batch &, const S_ &S, int64_t) : cell(S.cell), img(S.img) {
#pragma unroll
        for (int k = 0; k < 9; ++k) hi[k] = S.cell->hif[k];
    }
    template <typename S_> __device__ __forceinline__ void set(const S_ &S, int place) {
        x = S.px[place];
        y = S.py[place];
        z = S.pz[place];
    }
    template <typename S_>
    __device__ __forceinline__ void diff(const S_ &S, int j, int, double &dx, double &dy, double &dz) const {
        const double ex = x - S.px[j], ey = y - S.py[j], ez = z - S.pz[j];
        const float fx = f32_screen(ex), fy = f32_screen(ey), fz = f32_screen(ez);
        float n[3], w[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            w[r] = hi[r] * fx + hi[r + 3] * fy + hi[r + 6] * fz;
            n[r] = image_round(w[r]);
        }
        const float off = fmaxf(fabsf(w[0] - n[0]), fmaxf(fabsf(w[1] - n[1]), fabsf(w[2] - n[2])));
        const float big = fmaxf(fabsf(w[0]), fmaxf(fabsf(w[1]), fabsf(w[2])));
        dx = ex;
        dy = ey;
        dz = ez;
        if (off < 0.4999f && big < 1.5f) {
            const float kf = 9.f * n[0] + 3.f * n[1] + n[2];
            if (kf == 0.f) return;
            if (!img) {
                const double3 d = image_near(*cell, n[0], n[1], n[2], ex, ey, ez);
                dx = d.x;
                dy = d.y;
                dz = d.z;
                return;
            }
            const double *v = img + 3 * ((int)kf + 13);
            dx -= v[0];
            dy -= v[1];
            dz -= v[2];
        } else {
            const double3 d = min_image_far(*cell, ex, ey, ez);
            dx = d.x;
            dy = d.y;
            dz = d.z;
        }
    }
};

// ---------------------------------------------------------------------------
// EMT for G beads (b0 ..) of one trajectory, G <= emt_group.  Adds forces into B.f* (stores them
// when `store`), sets dens, adds the beads' energies into B.epot.  Must be called by all threads
// of the CTA.
//
// Atoms are staged by species: places [seg[0], seg[1]) of a bead hold the atoms of species slot 0,
// [seg[1], seg[2]) those of slot 1, the rest are not EMT; bead g follows at place g N.  Almost every pair has two atoms of
// the metal, so pairs are walked per species with the species' constants in registers and no
// branch; the few pairs of the two species run in a loop of their own (in one common walk nearly
// every warp met one of them, and took both branches).
//
// Pairs of one species, FP32 forces: a thread takes one atom i and a run of partners j and keeps
// its sums in registers; every pair is evaluated from both ends, in the density pass and again in
// the force pass (about 80 and 100 instructions).  Storing a pair's six values and reading them
// back by both ends took as many instructions and waited on the L2 for them.
// Pairs of one species, FP64 forces (M atoms): (i, j = (i+k) mod M), k = 1..M/2, in scratch slot
// (k-1) M + i (the k = M/2 row holds only i < M/2 when M is even).  A thread takes one atom i
// and a run of k: its side of a pair sums in registers, the other side is read back from the
// scratch by the thread that owns j (lanes hold consecutive i: every access coalesces).  A
// shared-memory FP64 addition costs 137 cycles a warp, reading the value back 5.
//   pass 1  distance, density term rho, pair energy, and the scalars q = -rho'/r, fv of the force
//   epilogue (per atom) sigma -> s, cohesive energy, embedded density, A = (dE/ds)/(beta eta2 sigma)
//   pass 2  cc = (A_i + A_j) q + fv, force += cc d on i; FP64: cc left in q's slot, then -cc d on j
// ---------------------------------------------------------------------------
static __device__ __forceinline__ const EmtPairs<double> &emt_pairs(const EmtConst &E, double) { return E.pd; }
static __device__ __forceinline__ const EmtPairs<float> &emt_pairs(const EmtConst &E, float) { return E.pf; }

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
    __device__ __forceinline__ void join(const EnergySum &o) { s += o.s; }
    __device__ __forceinline__ double value() const { return s; }
};
template <> struct EnergySum<float> {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = __fadd_rn(s, x), z = __fsub_rn(t, s);
        c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(x, z)));
        s = t;
    }
    __device__ __forceinline__ void join(const EnergySum &o) {
        add(o.s);
        c = __fadd_rn(c, o.c);
    }
    __device__ __forceinline__ double value() const { return f64_of(s) + f64_of(c); }
};

static __device__ __forceinline__ bool is_zero(double x) {
    return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}
static __device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
static __device__ __forceinline__ double wide(double x) { return x; }
static __device__ __forceinline__ double wide(float x) { return f64_of(x); }

// acc[place] += the sum of v over the lanes of each place (a warp's lanes hold one, or a few where
// it spans beads): one shared-memory addition per place.
template <typename R> static __device__ __forceinline__ void warp_add(R *acc, int place, R v) {
    for (unsigned left = 0xffffffffu; left;) {
        const int src = __ffs(left) - 1, pl = __shfl_sync(0xffffffffu, place, src);
        const bool mine = place == pl;
        R s = mine ? v : R(0);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 31) == src && !is_zero(s)) atomicAdd(&acc[pl], s);
        left &= ~__ballot_sync(0xffffffffu, mine);
    }
}

// Beyond the cutoff, like the reference's `if (r > cutoff*rcut) cycle` (pes_emt_mod.f90:660): a
// distance that is not a number enters the sums.  FP64: on the high words, the exact comparison
// only when they are equal.
static __device__ __forceinline__ bool beyond(double r2, double cut2) {
    const int a = __double2hiint(r2), c = __double2hiint(cut2);
    return a == c ? r2 > cut2 : a > c && a <= 0x7ff00000;
}
static __device__ __forceinline__ bool beyond(float r2, float cut2) { return r2 > cut2; }

// Runs per atom (1..16) of its `span` partners so that the G M C work items of the pair loops fill
// the CTA's rounds best (cost: rounds x run length; a run also pays its sums once).  One warp,
// lane = candidate.
static __device__ __forceinline__ int pair_chunks(int M, int span, int G, int nt) {
    const int C = (threadIdx.x & 15) + 1;
    const int64_t cost =
        C <= span || C == 1 ? (int64_t)((G * M * C + nt - 1) / nt) * (2 * ((span + C - 1) / C) + 1) : 1 << 26;
    const int best = __reduce_min_sync(0xffffffffu, (int)min(cost, (int64_t)1 << 26) << 4 | (C - 1));
    return (best & 15) + 1;
}

// One species' places in the staged beads (m0 .. m0 + M - 1 of each), the runs per atom and, FP64
// forces, the scratch records of its pairs: (d, q) at rec4 + 4 slot, (fv, rho) at rec2 + 2 slot,
// `stride` values per bead.
template <typename R> struct Species {
    int N, G, m0, M, C;
    R *rec4, *rec2;
    int64_t stride;
    R cut2;
};

// calls f(bead, atom, first, last) for this thread's runs; `span` partners per atom
template <typename F> static __device__ __forceinline__ void for_runs(int G, int M, int C, int span, F f) {
    const int per = (span + C - 1) / C, GM = G * M;
    for (int w = threadIdx.x; w < GM * C; w += blockDim.x) {
        const int c = w / GM, g = (w - c * GM) / M;
        f(g, w - c * GM - g * M, c * per, min((c + 1) * per, span));
    }
}

// ---- FP32 forces: pairs of one species from both ends -------------------------------------
static __device__ __forceinline__ void pairs_density(const SmemEmt<float> &S, PlaceDiff<float> &D, const PairK<float> &k,
                                                     const Species<float> &A, bool, EnergySum<float> &) {
    for_runs(A.G, A.M, A.C, A.M, [&](int g, int i, int j0, int j1) {
        const int gp = g * A.N + A.m0;
        float acc = 0.f;
        D.set(S, gp + i);
        for (int j = j0; j < j1; ++j) {
            float rx, ry, rz;
            D.diff(S, gp + j, A.N, rx, ry, rz);
            const float r2 = rx * rx + ry * ry + rz * rz;
            if (j != i && !beyond(r2, A.cut2)) {
                const float r = r2 * Math<float>::rsq(r2);
                float theta, rt1;
                emt_theta<float>(k.acut, k.rcut, r, theta, rt1);
                acc += k.g * (theta * Math<float>::ex(-k.eta * (r - k.b)));
            }
        }
        if (A.C == 1) S.sig[gp + i] = acc;
        else atomicAdd(&S.sig[gp + i], acc);
    });
}
static __device__ __forceinline__ void pairs_density_2(const SmemEmt<float> &, const Species<float> &) {}

// forces and pair energies (a pair's energy from its first end)
static __device__ __forceinline__ void pairs_force(const SmemEmt<float> &S, PlaceDiff<float> &D, const PairK<float> &k,
                                                   const Species<float> &A, bool do_forces, EnergySum<float> &e_pair) {
    for_runs(A.G, A.M, A.C, A.M, [&](int g, int i, int j0, int j1) {
        const int gp = g * A.N + A.m0;
        const float Ai = S.A[gp + i];
        float fx = 0.f, fy = 0.f, fz = 0.f;
        EnergySum<float> e_run;
        D.set(S, gp + i);
        for (int j = j0; j < j1; ++j) {
            float rx, ry, rz;
            D.diff(S, gp + j, A.N, rx, ry, rz);
            const float r2 = rx * rx + ry * ry + rz * rz;
            if (j != i && !beyond(r2, A.cut2)) {
                const float ir = Math<float>::rsq(r2), r = r2 * ir;
                float theta, rt1;
                emt_theta<float>(k.acut, k.rcut, r, theta, rt1);
                const float phi = theta * Math<float>::ex(-k.eta * (r - k.b));
                const float psi = theta * Math<float>::ex(-k.kb * (r - k.b));
                e_run.add(i < j ? -(k.c * psi) : 0.f);
                const float q = k.g * (k.etaq + rt1) * phi * ir, fv = -(k.c * (k.kb + rt1) * psi * ir);
                const float cc = Ai * q + S.A[gp + j] * q + fv;
                fx += cc * rx;
                fy += cc * ry;
                fz += cc * rz;
            }
        }
        if (do_forces) {
            atomicAdd(&S.fx[gp + i], fx);
            atomicAdd(&S.fy[gp + i], fy);
            atomicAdd(&S.fz[gp + i], fz);
        }
        if (A.G == 1) e_pair.join(e_run);
        else atomicAdd(&S.en[gp + i], e_run.value());
    });
}
static __device__ __forceinline__ void pairs_force_2(const SmemEmt<float> &, const Species<float> &) {}

// ---- FP64 forces: each pair once, its other end through the scratch ----------------------
static __device__ __forceinline__ void pairs_density(const SmemEmt<double> &S, PlaceDiff<double> &D,
                                                     const PairK<double> &k, const Species<double> &A, bool do_forces,
                                                     EnergySum<double> &e_pair) {
    const int M = A.M, K = M / 2;
    for_runs(A.G, M, A.C, K, [&](int g, int i, int k0, int k1) {
        const int gp = g * A.N + A.m0;
        double acc = 0.0;
        EnergySum<double> e_run;
        D.set(S, gp + i);
        if (2 * K == M && i >= K) k1 = min(k1, K - 1);  // the last row of an even M holds each pair once
        for (int kk = k0; kk < k1; ++kk) {
            int j = i + kk + 1;
            if (j >= M) j -= M;
            double q = 0.0, fv = 0.0, rho = 0.0, rx, ry, rz;
            D.diff(S, gp + j, A.N, rx, ry, rz);
            const double r2 = rx * rx + ry * ry + rz * rz;
            if (!beyond(r2, A.cut2)) {
                const double ir = Math<double>::rsq(r2), r = r2 * ir;
                double theta, rt1;
                emt_theta<double>(k.acut, k.rcut, r, theta, rt1);
                const double phi = theta * Math<double>::ex(-k.eta * (r - k.b));
                const double psi = theta * Math<double>::ex(-k.kb * (r - k.b));
                rho = k.g * phi;
                acc += rho;
                e_run.add(-(k.c * psi));
                q = (k.etaq + rt1) * rho * ir;
                fv = -(k.c * (k.kb + rt1) * psi * ir);
            }
            const int64_t slot = A.stride * g + kk * M + i;
            *reinterpret_cast<double2 *>(A.rec2 + 2 * slot) = make_double2(fv, rho);
            if (do_forces) {
                double2 *p = reinterpret_cast<double2 *>(A.rec4 + 4 * slot);
                p[0] = make_double2(rx, ry);
                p[1] = make_double2(rz, q);
            }
        }
        if (A.C == 1) S.sig[gp + i] = acc;
        else atomicAdd(&S.sig[gp + i], acc);
        if (A.G == 1) e_pair.join(e_run);
        else if (A.C == 1) S.en[gp + i] = e_run.value();
        else atomicAdd(&S.en[gp + i], e_run.value());
    });
}

// the densities' other end
static __device__ __forceinline__ void pairs_density_2(const SmemEmt<double> &S, const Species<double> &A) {
    const int M = A.M, K = M / 2;
    for_runs(A.G, M, A.C, K, [&](int g, int j, int k0, int k1) {
        double acc = 0.0;
        // row k holds the pair whose second atom is j at place j - k (mod M); the last row of an
        // even M only for places below K
        if (2 * K == M && k1 == K && j < K) k1 = K - 1;
#pragma unroll 4
        for (int kk = k0; kk < k1; ++kk) {
            int m = j - kk - 1;
            if (m < 0) m += M;
            const double rho = A.rec2[2 * (A.stride * g + kk * M + m) + 1];
            if (!is_zero(rho)) acc += rho;
        }
        if (A.C == 1) S.sig[g * A.N + A.m0 + j] += acc;
        else atomicAdd(&S.sig[g * A.N + A.m0 + j], acc);
    });
}

static __device__ __forceinline__ void pairs_force(const SmemEmt<double> &S, PlaceDiff<double> &, const PairK<double> &,
                                                   const Species<double> &A, bool do_forces, EnergySum<double> &) {
    if (!do_forces) return;
    const int M = A.M, K = M / 2;
    for_runs(A.G, M, A.C, K, [&](int g, int i, int k0, int k1) {
        const int gp = g * A.N + A.m0;
        const double Ai = S.A[gp + i];
        double fx = 0.0, fy = 0.0, fz = 0.0;
        if (2 * K == M && i >= K) k1 = min(k1, K - 1);
#pragma unroll 2
        for (int kk = k0; kk < k1; ++kk) {
            int j = i + kk + 1;
            if (j >= M) j -= M;
            const int64_t slot = A.stride * g + kk * M + i;
            double2 *p = reinterpret_cast<double2 *>(A.rec4 + 4 * slot);
            const double2 a = p[0], c = p[1];
            if (is_zero(c.y)) continue;  // beyond the cutoff: the 0 stays in q's place
            const double cc = (Ai + S.A[gp + j]) * c.y + A.rec2[2 * slot];
            A.rec4[4 * slot + 3] = cc;
            fx += cc * a.x;
            fy += cc * a.y;
            fz += cc * c.x;
        }
        if (A.C == 1) {
            S.fx[gp + i] = fx;
            S.fy[gp + i] = fy;
            S.fz[gp + i] = fz;
        } else {
            atomicAdd(&S.fx[gp + i], fx);
            atomicAdd(&S.fy[gp + i], fy);
            atomicAdd(&S.fz[gp + i], fz);
        }
    });
}

// the forces' other end
static __device__ __forceinline__ void pairs_force_2(const SmemEmt<double> &S, const Species<double> &A) {
    const int M = A.M, K = M / 2;
    for_runs(A.G, M, A.C, K, [&](int g, int j, int k0, int k1) {
        double fx = 0.0, fy = 0.0, fz = 0.0;
        if (2 * K == M && k1 == K && j < K) k1 = K - 1;
#pragma unroll 2
        for (int kk = k0; kk < k1; ++kk) {
            int m = j - kk - 1;
            if (m < 0) m += M;
            const double2 *p = reinterpret_cast<const double2 *>(A.rec4 + 4 * (A.stride * g + kk * M + m));
            const double2 a = p[0], c = p[1];
            if (is_zero(c.y)) continue;
            fx -= c.y * a.x;
            fy -= c.y * a.y;
            fz -= c.y * c.x;
        }
        const int i = g * A.N + A.m0 + j;
        if (A.C == 1) {
            S.fx[i] += fx;
            S.fy[i] += fy;
            S.fz[i] += fz;
        } else {
            atomicAdd(&S.fx[i], fx);
            atomicAdd(&S.fy[i], fy);
            atomicAdd(&S.fz[i], fz);
        }
    });
}

template <typename R>
static __device__ void emt_beads(const Batch &B, const EmtConst &E, const SmemEmt<R> &S, int t, int b0, int G,
                                 bool do_forces, bool store = false) {
    const int N = B.natoms[t], GN = G * N;
    const int64_t base = B.ba_off[t] + (int64_t)b0 * N;
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
    for (int p = tid; p < GN; p += nt) {
        const int g0 = p / N * N;
        const int64_t k = base + g0 + S.perm[p - g0];
        const double x = B.rx[k], y = B.ry[k], z = B.rz[k];
        if constexpr (sizeof(R) == 4) {
            float hi[3], lo[3];
            split3(x, y, z, hi, lo);
            S.ph[p] = make_float4(hi[0], hi[1], hi[2], 0.f);
            S.pl[p] = make_float4(lo[0], lo[1], lo[2], 0.f);
        } else {
            S.px[p] = x;
            S.py[p] = y;
            S.pz[p] = z;
        }
        S.sig[p] = R(0);
        S.A[p] = R(0);
        S.fx[p] = R(0);
        S.fy[p] = R(0);
        S.fz[p] = R(0);
        if (G > 1) S.en[p] = 0.0;
    }
    if (tid < 32) {
        const int m0 = S.seg[1], m1 = S.seg[2] - m0;
        const int c0 = pair_chunks(m0, sizeof(R) == 8 ? m0 / 2 : m0, G, nt),
                  c1 = pair_chunks(m1, sizeof(R) == 8 ? m1 / 2 : m1, G, nt);
        if (tid == 0) {
            S.seg[4] = c0;
            S.seg[5] = c1;
        }
    }
    __syncthreads();
    const int n0 = S.seg[1], n1 = S.seg[2] - S.seg[1];

    const int NK = N * (N / 2);
    R *const rec4 = (R *)B.pair_scratch + 6 * (B.pair_off[t] + (int64_t)b0 * NK), *const rec2 = rec4 + 4 * (int64_t)G * NK;
    const EmtPairs<R> &Q = emt_pairs(E, R(0));
    const R cut2 = Q.cut2;
    PlaceDiff<R> D(B, S, base);
    EnergySum<R> e_pair;  // one bead: this thread's pair energies
    // calls f(constants, places) for each species that has pairs
    auto each_species = [&](auto f) {
        for (int s = 0, off = 0; s < E.nspecies; ++s) {
            const int m0 = S.seg[s], M = S.seg[s + 1] - m0;
            if (M < 2) continue;
            const PairK<R> k{Q.acut, Q.rcut, Q.eta[s], Q.etaq[s], Q.b[s], Q.kb[s], Q.g[s], Q.c[s]};
            const Species<R> A{N, G, m0, M, S.seg[4 + s], rec4 + 4 * off, rec2 + 2 * off, NK, cut2};
            f(k, A);
            off += M * (M - 1) / 2;
        }
    };

    // ---- pass 1, pairs of one species -------------------------------------------------
    each_species([&](const PairK<R> &k, const Species<R> &A) { pairs_density(S, D, k, A, do_forces, e_pair); });
    // ---- pass 1, pairs of the two species: a warp's lanes over the slot-1 atoms ----------
    const int t0 = E.type_of_slot[0], t1 = E.type_of_slot[1];
    const int xoff = n0 * (n0 - 1) / 2 + n1 * (n1 - 1) / 2;  // cross pairs follow in the scratch
    const bool cross = n0 > 0 && n1 > 0;
    __syncthreads();
    if (cross) {
        const R acut = Q.acut, rcut = Q.rcut, eta0 = Q.eta[0], eta1 = Q.eta[1], bs0 = Q.b[0], bs1 = Q.b[1],
                kb0 = Q.kb[0], kb1 = Q.kb[1], gaj = Q.gx[0], gja = Q.gx[1], caj = Q.cx[0], cja = Q.cx[1];
        // work items (bead, slot-1 atom), walked in whole warps: each item meets the bead's slot-0 atoms
        const int items = G * n1;
        for (int w0 = tid & ~31; w0 < items; w0 += nt) {
            const int w = w0 + (tid & 31);
            const bool on = w < items;
            const int g = on ? w / n1 : G - 1, jj = on ? w - g * n1 : 0;
            const int j = g * N + n0 + jj;
            for (int a = 0; a < n0; ++a) {
                R sa = R(0);
                EnergySum<R> e_run;
                if (on) {
                    R q_a = R(0), q_j = R(0), fv = R(0), rx = R(0), ry = R(0), rz = R(0);
                    // pes(ti, tj) of the pair's first atom in the (i, i+k mod N) order, should the table
                    // not be symmetric
                    const int ia = S.perm[a], ij = S.perm[n0 + jj], d = ij - ia, dk = d > 0 ? d : d + N;
                    const bool a_first = 2 * dk < N || (2 * dk == N && ia < ij);
                    if ((E.pair_mask >> (a_first ? t0 * kMaxTypes + t1 : t1 * kMaxTypes + t0)) & 1u) {
                        D.set(S, g * N + a);
                        D.diff(S, j, N, rx, ry, rz);
                        const R r2 = rx * rx + ry * ry + rz * rz;
                        if (!beyond(r2, cut2)) {
                            const R ir = Math<R>::rsq(r2), r = r2 * ir;
                            R theta, rt1;
                            emt_theta<R>(acut, rcut, r, theta, rt1);
                            const R phi_j = theta * Math<R>::ex(-eta1 * (r - bs1));
                            const R psi_j = theta * Math<R>::ex(-kb1 * (r - bs1));
                            const R phi_a = theta * Math<R>::ex(-eta0 * (r - bs0));
                            const R psi_a = theta * Math<R>::ex(-kb0 * (r - bs0));
                            sa = gaj * phi_j;
                            S.sig[j] += gja * phi_a;  // this thread alone owns j here
                            e_run.add(-R(0.5) * (caj * psi_j + cja * psi_a));
                            fv = -R(0.5) * (caj * (kb1 + rt1) * psi_j + cja * (kb0 + rt1) * psi_a) * ir;
                            q_a = gaj * (eta1 + rt1) * phi_j * ir;
                            q_j = gja * (eta0 + rt1) * phi_a * ir;
                        }
                    }
                    if (do_forces) {
                        const int64_t slot = (int64_t)NK * g + xoff + a * n1 + jj;
                        R *const p = rec4 + 4 * slot, *const p2 = rec2 + 2 * slot;
                        p[0] = rx;
                        p[1] = ry;
                        p[2] = rz;
                        p[3] = q_a;
                        p2[0] = fv;
                        p2[1] = q_j;
                    }
                    if (G == 1) e_pair.join(e_run);
                    else S.en[j] += e_run.value();  // this thread alone owns j here
                }
                warp_add<R>(S.sig, g * N + a, sa);
            }
        }
    }
    __syncthreads();
    each_species([&](const PairK<R> &, const Species<R> &A) { pairs_density_2(S, A); });
    __syncthreads();

    // ---- per-atom epilogue ---------------------------------------------------
    double e_atom = 0.0;
    const int ne = n0 + n1;
    for (int w = tid; w < G * ne; w += nt) {
        const int g = w / ne, p = w - g * ne, i = g * N + p;
        const int s = p >= n0;
        double sc = (double)S.sig[i], cl = sc;
        // above 1e-9 (by its high word) neither floor of pes_emt_mod.f90:793 acts
        if (__double2hiint(sc) <= 0x3e112e0b || __double2hiint(sc) >= 0x7ff00000) {
            sc = fmax((double)1e-30f, sc);  // single-precision 1e-30
            cl = fmax(kTolerance, sc);
        }
        const double be = E.betaeta2[s], sa = div_by(-log(cl * kTwelfth), be, E.ibe[s]);
        const double lsa = E.lambda[s] * sa, el = exp_t64(-lsa), ek = exp_t64(-E.kappa[s] * sa);
        const double e = E.e0[s] * (fma(lsa, el, el) - 1.0) + E.v6[s] * ek;
        const double bs = be * sc;
        S.A[i] = (R)div_by(E.e0l2[s] * sa * el + E.v6k[s] * ek, bs, rcp_nr(bs));
        B.dens[base + g * N + S.perm[p]] = E.n0[s] * exp_t64(E.dens_exp[s] * sa);
        if (G == 1) e_atom += e;
        else S.en[i] += e;
    }
    __syncthreads();

    // ---- pass 2 ----------------------------------------------------------------------
    if (do_forces || sizeof(R) == 4)
        each_species([&](const PairK<R> &k, const Species<R> &A) { pairs_force(S, D, k, A, do_forces, e_pair); });
    if (G == 1) {
        const double etot = block_sum(e_pair.value() + e_atom, S.red);  // contains __syncthreads
        if (tid == 0) B.epot[B.bead_off[t] + b0] += etot;
    } else {
        __syncthreads();
        for (int g = tid >> 5; g < G; g += nt >> 5) {  // a warp per bead
            double e = 0.0;
            for (int i = tid & 31; i < ne; i += 32) e += S.en[g * N + i];
            for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if ((tid & 31) == 0) B.epot[B.bead_off[t] + b0 + g] += e;
        }
    }
    if (!do_forces) {
        __syncthreads();
        return;
    }
    if (cross) {  // pairs of the two species
        const int items = G * n1;
        for (int w0 = tid & ~31; w0 < items; w0 += nt) {
            const int w = w0 + (tid & 31);
            const bool on = w < items;
            const int g = on ? w / n1 : G - 1, jj = on ? w - g * n1 : 0;
            const int j = g * N + n0 + jj;
            for (int a = 0; a < n0; ++a) {
                R gx = R(0), gy = R(0), gz = R(0);
                if (on) {
                    const int64_t slot = (int64_t)NK * g + xoff + a * n1 + jj;
                    const R *const p = rec4 + 4 * slot, *const p2 = rec2 + 2 * slot;
                    const R cc = S.A[g * N + a] * p[3] + S.A[j] * p2[1] + p2[0];
                    gx = cc * p[0];
                    gy = cc * p[1];
                    gz = cc * p[2];
                    S.fx[j] -= gx;  // this thread alone owns j here
                    S.fy[j] -= gy;
                    S.fz[j] -= gz;
                }
                warp_add<R>(S.fx, g * N + a, gx);
                warp_add<R>(S.fy, g * N + a, gy);
                warp_add<R>(S.fz, g * N + a, gz);
            }
        }
    }
    __syncthreads();
    each_species([&](const PairK<R> &, const Species<R> &A) { pairs_force_2(S, A); });
    __syncthreads();
    for (int p = tid; p < GN; p += nt) {
        const int g0 = p / N * N;
        const int64_t k = base + g0 + S.perm[p - g0];
        const double fx = wide(S.fx[p]), fy = wide(S.fy[p]), fz = wide(S.fz[p]);
        if (store) {
            B.fx[k] = fx;
            B.fy[k] = fy;
            B.fz[k] = fz;
        } else {
            B.fx[k] += fx;
            B.fy[k] += fy;
            B.fz[k] += fz;
        }
    }
    __syncthreads();
}

}  // namespace mdt
