// mdt_acsf.cuh -- atom-centred symmetry functions as CTA/warp device functions, shared by
// the HDNNP/surrogate force kernels (mdt_nn_kernels.cuh) and the training kernels (mdt_train.cu).
//
// One warp owns one central atom i.  Its neighbour cache (per neighbour q: the vector
// d_q = x_q - x_i, r_q, fc(r_q), dfc/dr(r_q) and exp(-eta r_q^2) for every distinct G3 eta
// of the element) lives in the warp's shared memory.  Triplets (j<k) are walked with a
// lane-strided flat index over the upper triangle.  Three walks exist:
//   forward  G_s                         (atomsymfunction2.f90:80-170, atomsymfunction3Andi.f90:90-257)
//   VJP      F -= sum_s c_s dG_s/dx       (forces from c_s = dE/dG_s)
//   JVP      v_s = sum_k u_k . (-dG_s/dx_k) (the force-loss adjoint for training)
// The G3 derivative factors p1, p2, p3 are those of atomsymfunction3Andi.f90:209-222.
// For the VJP they are summed over functions in factored form: with
// u_s = c_s 2^(1-zeta) (1+lambda cos)^(zeta-1) exp(-eta sum r^2),
//   P1 = pfc (1/(r_ij r_ik) - cos/r_ij^2) A1 - 2 pfc A2 + fc_ik fc_jk dfc_ij/r_ij A3
//   P2 = pfc (1/(r_ij r_ik) - cos/r_ik^2) A1 - 2 pfc A2 + fc_ij fc_jk dfc_ik/r_ik A3
//   P3 = pfc/(r_ij r_ik) A1 + 2 pfc A2 - fc_ij fc_ik dfc_jk/r_jk A3
// where A1 = sum u_s zeta_s lambda_s, A2 = sum u_s eta_s (1+lambda_s cos), A3 = sum u_s (1+lambda_s cos):
// three multiply-adds per function and triplet instead of three full derivative factors.
#pragma once
#include <type_traits>

#include "mdt_common.cuh"
#include "mdt_nn.cuh"

namespace mdt {

constexpr int kMaxG3 = 24;  // G3 functions per element held in lane registers
constexpr double kAng2BohrD = 1.0 / kBohr2Ang;

template <typename R> struct WarpCache {
    R *nb;          // [q][stride]
    R *slotf;       // [q][3]
    int *nbatom;    // [q]
    int8_t *nbelem; // [q]
    int st;
};

template <typename R> __device__ __forceinline__ R warp_sum(R v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Triangle walk over neighbour pairs (q3 < q4): lane-strided flat index, advanced by 32
// pairs per iteration without a square-root decode.
struct TriWalk {
    int q3, q4, n;
    bool valid;
    __device__ __forceinline__ void init(int cnt, int lane) {
        n = cnt;
        q3 = 0;
        q4 = 1 + lane;
        normalize();
    }
    __device__ __forceinline__ void normalize() {
        while (q3 < n - 1 && q4 >= n) {
            const int over = q4 - n;
            ++q3;
            q4 = q3 + 1 + over;
        }
        valid = q3 < n - 1 && q4 < n;
    }
    __device__ __forceinline__ void next() {
        q4 += 32;
        normalize();
    }
};

// Balanced row walk over the same triangle: lane L owns the row pairs (r, nrows-1-r)
// for r = L, L+32, ...; each pair holds cnt pairs (q3, q4) in total, so every lane runs
// the same number of iterations, and because a lane keeps its row q3 for many
// iterations, the q3 side of a triplet can be accumulated in registers (flushed when
// the row changes) while the q4 sides of the 32 lanes are distinct atoms.
struct RowWalk {
    int cnt, nrows, p, it, len0, q3, q4;
    bool valid, row_end;  // row_end: q3 changes after this triplet
    __device__ __forceinline__ void init(int c, int lane) {
        cnt = c;
        nrows = c - 1;
        p = lane;
        start();
    }
    __device__ __forceinline__ void start() {
        it = 0;
        const int npairs = (nrows + 1) / 2;
        valid = p < npairs;
        if (!valid) return;
        len0 = nrows - p;  // row p holds q4 = p+1 .. cnt-1
        set();
    }
    __device__ __forceinline__ int total() const { return (nrows - 1 - p == p) ? len0 : cnt; }
    __device__ __forceinline__ void set() {
        if (it < len0) {
            q3 = p;
            q4 = p + 1 + it;
        } else {
            q3 = nrows - 1 - p;
            q4 = q3 + 1 + (it - len0);
        }
        row_end = (it == len0 - 1) || (it == total() - 1);
    }
    __device__ __forceinline__ void next() {
        ++it;
        if (it >= total()) {
            p += 32;
            start();
            return;
        }
        set();
    }
};

__device__ __forceinline__ int pack_nb(int j, int n1, int n2, int n3) {
    return j | ((n1 + 8) << 16) | ((n2 + 8) << 20) | ((n3 + 8) << 24);
}

// lattice rows (bohr) and the inverse of the column matrix, without fused operations so
// that the cell folding matches the oracle bit for bit.  box: 9 doubles column major (A).
static __device__ void acsf_lattice(const double *bx, double *lat) {
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) lat[3 * i + k] = __dmul_rn(bx[3 * i + k], kAng2BohrD);
    double A[9];
    for (int i = 0; i < 3; ++i)
        for (int k = 0; k < 3; ++k) A[k * 3 + i] = lat[3 * i + k];
    double *I = lat + 9;
    auto m = [](double a, double b2) { return __dmul_rn(a, b2); };
    auto sb = [](double a, double b2) { return __dsub_rn(a, b2); };
    const double det = __dadd_rn(__dsub_rn(m(A[0], sb(m(A[4], A[8]), m(A[5], A[7]))),
                                            m(A[1], sb(m(A[3], A[8]), m(A[5], A[6])))),
                                 m(A[2], sb(m(A[3], A[7]), m(A[4], A[6]))));
    I[0] = __ddiv_rn(sb(m(A[4], A[8]), m(A[5], A[7])), det);
    I[1] = __ddiv_rn(sb(m(A[2], A[7]), m(A[1], A[8])), det);
    I[2] = __ddiv_rn(sb(m(A[1], A[5]), m(A[2], A[4])), det);
    I[3] = __ddiv_rn(sb(m(A[5], A[6]), m(A[3], A[8])), det);
    I[4] = __ddiv_rn(sb(m(A[0], A[8]), m(A[2], A[6])), det);
    I[5] = __ddiv_rn(sb(m(A[2], A[3]), m(A[0], A[5])), det);
    I[6] = __ddiv_rn(sb(m(A[3], A[7]), m(A[4], A[6])), det);
    I[7] = __ddiv_rn(sb(m(A[1], A[6]), m(A[0], A[7])), det);
    I[8] = __ddiv_rn(sb(m(A[0], A[4]), m(A[1], A[3])), det);
}

// positions A -> bohr, folded into the cell (RuNNer_src/translate.f90)
static __device__ __forceinline__ void acsf_wrap_one(double xa, double ya, double za, const double *lat, double &x,
                                                     double &y, double &z) {
    x = __dmul_rn(xa, kAng2BohrD);
    y = __dmul_rn(ya, kAng2BohrD);
    z = __dmul_rn(za, kAng2BohrD);
    const double *I = lat + 9;
    double f[3];
    for (int d = 0; d < 3; ++d)
        f[d] = __dadd_rn(__dadd_rn(__dmul_rn(I[3 * d], x), __dmul_rn(I[3 * d + 1], y)), __dmul_rn(I[3 * d + 2], z));
    for (int d = 0; d < 3; ++d) {
        const double s = floor(f[d]);
        if (s != 0.0) {
            x = __dsub_rn(x, __dmul_rn(s, lat[3 * d]));
            y = __dsub_rn(y, __dmul_rn(s, lat[3 * d + 1]));
            z = __dsub_rn(z, __dmul_rn(s, lat[3 * d + 2]));
        }
    }
}

// the oracle's cutoff test of one image in FP64, in its operation order (no fused multiply-add)
static __device__ __noinline__ bool acsf_inside(double xi, double yi, double zi, double xj, double yj, double zj,
                                                double d1n, double d2n, double d3n, const double *L, double cut2) {
    const double xt = __dadd_rn(__dadd_rn(__dadd_rn(xj, __dmul_rn(d1n, L[0])), __dmul_rn(d2n, L[3])),
                                __dmul_rn(d3n, L[6]));
    const double yt = __dadd_rn(__dadd_rn(__dadd_rn(yj, __dmul_rn(d1n, L[1])), __dmul_rn(d2n, L[4])),
                                __dmul_rn(d3n, L[7]));
    const double zt = __dadd_rn(__dadd_rn(__dadd_rn(zj, __dmul_rn(d1n, L[2])), __dmul_rn(d2n, L[5])),
                                __dmul_rn(d3n, L[8]));
    const double e1 = __dsub_rn(xt, xi), e2 = __dsub_rn(yt, yi), e3 = __dsub_rn(zt, zi);
    return __dadd_rn(__dadd_rn(__dmul_rn(e1, e1), __dmul_rn(e2, e2)), __dmul_rn(e3, e3)) <= cut2;
}

// neighbour list of atom i in RuNNer's order (neighbor_para_short.f90:117-163).
// Returns the count (may exceed maxnb: the caller flags the overflow).  An FP32 screen, the exact
// FP64 test only within 1e-4 (relative) of the cutoff.  Three FP64 subtractions per atom j; formed
// per image, with the cell's conversions, the screen was 15 FP64-pipe instructions for each of
// an atom's 27 and more images: most of the generic FP32 kernel's FP64 work.
static __device__ int acsf_neighbors_one(const NNDev &M, int i, int N, const double *px, const double *py,
                                         const double *pz, const double *L, int na, int nbi, int nc, int *out) {
    const double cut2 = __dmul_rn(M.maxcut, M.maxcut);
    const float c2 = f32_screen(cut2), cut2f_hi = c2 * 1.0001f, cut2f_lo = c2 * 0.9999f;
    float Lf[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) Lf[k] = f32_screen(L[k]);
    int cnt = 0;
    const double xi = px[i], yi = py[i], zi = pz[i];
    for (int j = 0; j < N; ++j) {
        const double xj = px[j], yj = py[j], zj = pz[j];
        const float dx = f32_screen(xj - xi), dy = f32_screen(yj - yi), dz = f32_screen(zj - zi);
        for (int n1 = -na; n1 <= na; ++n1)
            for (int n2 = -nbi; n2 <= nbi; ++n2) {
                const float g1 = (float)n1, g2 = (float)n2;
                const float fx0 = dx + g1 * Lf[0] + g2 * Lf[3], fy0 = dy + g1 * Lf[1] + g2 * Lf[4],
                            fz0 = dz + g1 * Lf[2] + g2 * Lf[5];
                for (int n3 = -nc; n3 <= nc; ++n3) {
                    if (n1 == 0 && n2 == 0 && n3 == 0 && i == j) continue;
                    const float g3 = (float)n3;
                    const float fx = fx0 + g3 * Lf[6], fy = fy0 + g3 * Lf[7], fz = fz0 + g3 * Lf[8];
                    const float rf = fx * fx + fy * fy + fz * fz;
                    if (rf > cut2f_hi) continue;
                    if (rf < cut2f_lo || acsf_inside(xi, yi, zi, xj, yj, zj, n1, n2, n3, L, cut2)) {
                        if (cnt < M.maxnb) out[cnt] = pack_nb(j, n1, n2, n3);
                        ++cnt;
                    }
                }
            }
    }
    return cnt;
}

template <typename R> __device__ __forceinline__ R narrow(double x) {
    if constexpr (sizeof(R) == 4) return f32_of(x);
    else return x;
}

// neighbour cache of central atom i for its warp
template <typename R>
__device__ void acsf_cache(const NNDev &M, const WarpCache<R> &C, int i, int ei, int cnt, const int *words,
                           const double *px, const double *py, const double *pz, const int8_t *elem, const double *L) {
    const int lane = threadIdx.x & 31;
    const CutK<R> ck = cut_k<R>(M, ei);
    const R rc = ck.rc;
    const int ng = M.ng3eta[ei];
    for (int q = lane; q < cnt; q += 32) {
        const int w = words[q];
        const int j = w & 0xFFFF;
        const double n1 = f64_of((float)(((w >> 16) & 15) - 8)), n2 = f64_of((float)(((w >> 20) & 15) - 8)),
                     n3 = f64_of((float)(((w >> 24) & 15) - 8));
        const double dx = px[j] + n1 * L[0] + n2 * L[3] + n3 * L[6] - px[i];
        const double dy = py[j] + n1 * L[1] + n2 * L[4] + n3 * L[7] - py[i];
        const double dz = pz[j] + n1 * L[2] + n2 * L[5] + n3 * L[8] - pz[i];
        double ir;
        const R r = narrow<R>(dist_of(dx * dx + dy * dy + dz * dz, ir));
        R *e = C.nb + q * C.st;
        e[0] = narrow<R>(dx);
        e[1] = narrow<R>(dy);
        e[2] = narrow<R>(dz);
        e[3] = r;
        R fc = R(0), dfc = R(0);
        if (r <= rc) cutoff_fn<R>(M, ck, r, fc, dfc);
        e[4] = fc;
        e[5] = dfc;
        for (int m = 0; m < ng; ++m) e[6 + m] = NM<R>::ex(-g3_eta<R>(M, ei, m) * r * r);
        C.nbatom[q] = j;
        C.nbelem[q] = elem[j];
        C.slotf[3 * q] = R(0);
        C.slotf[3 * q + 1] = R(0);
        C.slotf[3 * q + 2] = R(0);
    }
    __syncwarp();
}

// G3 functions of an element, in SF order
struct G3List {
    int n;
    int idx[kMaxG3];
};

__device__ __forceinline__ G3List g3_list(const NNDev &M, int ei) {
    G3List g;
    g.n = 0;
    const int nsf = M.nsf[ei], sfb = ei * M.maxsf;
    for (int s = 0; s < nsf && g.n < kMaxG3; ++s)
        if (M.sftype[sfb + s] == 3) g.idx[g.n++] = s;
    return g;
}

// Per-triplet geometry shared by the three walks.
template <typename R> struct Triplet {
    const R *a, *c;  // cache rows of j and k
    R jx, jy, jz;    // d_j - d_k = x_j - x_k
    R rjk2, rjk, ijk, fcjk, dfcjk, rinv0, cost0, pfc;  // (ijk = 1/rjk: grid form, FP64)
    R ejk[kMaxEta];
};

template <typename R>
__device__ __forceinline__ bool triplet_setup(const NNDev &M, const WarpCache<R> &C, int ei, int q3, int q4,
                                              const CutK<R> &ck, Triplet<R> &T) {
    const R rc = ck.rc;
    T.a = C.nb + q3 * C.st;
    T.c = C.nb + q4 * C.st;
    if (!(T.a[3] <= rc && T.c[3] <= rc)) return false;
    T.jx = T.a[0] - T.c[0];
    T.jy = T.a[1] - T.c[1];
    T.jz = T.a[2] - T.c[2];
    T.rjk2 = T.jx * T.jx + T.jy * T.jy + T.jz * T.jz;
    if (!(T.rjk2 <= rc * rc)) return false;
    T.rjk = NM<R>::sq(T.rjk2);
    cutoff_fn<R>(M, ck, T.rjk, T.fcjk, T.dfcjk);
    T.rinv0 = NM<R>::rc(T.a[3] * T.c[3]);
    T.cost0 = (T.a[0] * T.c[0] + T.a[1] * T.c[1] + T.a[2] * T.c[2]) * T.rinv0;
    T.pfc = T.a[4] * T.c[4] * T.fcjk;
    const int ng = M.ng3eta[ei];
    for (int m = 0; m < ng; ++m) T.ejk[m] = NM<R>::ex(-g3_eta<R>(M, ei, m) * T.rjk2);
    return true;
}

__device__ __forceinline__ bool g3_match(const NNDev &M, int k, int ej, int ek) {
    const int e1 = M.e1[k], e2 = M.e2[k];
    return (e1 == ej && e2 == ek) || (e2 == ej && e1 == ek);
}

// (1 + lambda cos)^(zeta-1) exp(-eta sum r^2) 2^(1-zeta); returns false when 1+lambda cos <= 0
template <typename R>
__device__ __forceinline__ bool g3_term(const NNDev &M, int k, const Triplet<R> &T, R &plam, R &fgn) {
    plam = R(1) + (R)M.lam[k] * T.cost0;
    if (plam <= R(0)) return false;
    const int m = M.etaslot[k];
    const R pexp = T.a[6 + m] * T.c[6 + m] * T.ejk[m];
    const int iz = M.izeta[k];
    fgn = (iz >= 0 ? ipow<R>(plam, iz) : NM<R>::pw(plam, (R)M.zeta[k] - R(1))) * pexp * (R)M.pnorm[k];
    return true;
}

// grid-form G3 walks, defined at the end of this file
template <typename R> __device__ void acsf_g3_forward_fast(const NNDev &M, const WarpCache<R> &C, int ei, int cnt,
                                                           R *G);
template <typename R>
__device__ void acsf_g3_vjp_fast(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, const R *c, R &fix, R &fiy,
                                 R &fiz);
template <typename R>
__device__ void acsf_g3_jvp_fast(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, int i, const R *ux,
                                 const R *uy, const R *uz, R *v);

// ---- forward ------------------------------------------------------------------------
template <typename R> __device__ void acsf_forward(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, R *G) {
    const int lane = threadIdx.x & 31;
    const CutK<R> ck = cut_k<R>(M, ei);
    const R rc = ck.rc;
    const int nsf = M.nsf[ei], sfb = ei * M.maxsf;
    for (int s = 0; s < nsf; ++s) {
        if (M.sftype[sfb + s] != 2) continue;
        const R eta = sf_eta<R>(M, sfb + s), rs = sf_rs<R>(M, sfb + s);
        const int e1 = M.e1[sfb + s];
        R acc = R(0);
        for (int q = lane; q < cnt; q += 32) {
            const R *e = C.nb + q * C.st;
            if (C.nbelem[q] != e1 || !(e[3] <= rc)) continue;
            acc += NM<R>::ex(-eta * (e[3] - rs) * (e[3] - rs)) * e[4];
        }
        acc = warp_sum(acc);
        if (lane == 0) G[s] = acc;
    }
    if (M.ng3eta[ei] == 0) {  // no angular functions: no triplets to walk
        __syncwarp();
        return;
    }
    if (M.g3fast[ei]) {
        acsf_g3_forward_fast<R>(M, C, ei, cnt, G);
        return;
    }
    const G3List g3 = g3_list(M, ei);
    R acc[kMaxG3];
#pragma unroll
    for (int u = 0; u < kMaxG3; ++u) acc[u] = R(0);
    TriWalk tw;
    tw.init(cnt, lane);
    while (tw.valid) {
        Triplet<R> T;
        if (triplet_setup<R>(M, C, ei, tw.q3, tw.q4, ck, T)) {
            const int ej = C.nbelem[tw.q3], ek = C.nbelem[tw.q4];
#pragma unroll
            for (int u = 0; u < kMaxG3; ++u) {
                if (u >= g3.n) break;
                const int k = sfb + g3.idx[u];
                if (!g3_match(M, k, ej, ek)) continue;
                R plam, fgn;
                if (g3_term<R>(M, k, T, plam, fgn)) acc[u] += fgn * plam * T.pfc;
            }
        }
        tw.next();
    }
#pragma unroll
    for (int u = 0; u < kMaxG3; ++u) {
        if (u >= g3.n) break;
        const R v = warp_sum(acc[u]);
        if (lane == 0) G[g3.idx[u]] = v;
    }
    __syncwarp();
}

// ---- VJP: slot forces -= c . dG/dx; returns the central atom's force (all lanes) --------
template <typename R>
__device__ void acsf_vjp(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, const R *c, R &fix, R &fiy,
                         R &fiz) {
    const int lane = threadIdx.x & 31;
    const CutK<R> ck = cut_k<R>(M, ei);
    const R rc = ck.rc;
    const int nsf = M.nsf[ei], sfb = ei * M.maxsf;
    fix = fiy = fiz = R(0);
    for (int q = lane; q < cnt; q += 32) {
        const R *e = C.nb + q * C.st;
        if (!(e[3] <= rc)) continue;
        R dsum = R(0);
        for (int s = 0; s < nsf; ++s) {
            if (M.sftype[sfb + s] != 2 || C.nbelem[q] != M.e1[sfb + s]) continue;
            const R eta = sf_eta<R>(M, sfb + s), rs = sf_rs<R>(M, sfb + s);
            const R ex = NM<R>::ex(-eta * (e[3] - rs) * (e[3] - rs));
            dsum += c[s] * (R(-2) * eta * (e[3] - rs) * ex * e[4] + ex * e[5]);
        }
        const R fr = dsum / e[3];
        C.slotf[3 * q] -= fr * e[0];
        C.slotf[3 * q + 1] -= fr * e[1];
        C.slotf[3 * q + 2] -= fr * e[2];
        fix += fr * e[0];
        fiy += fr * e[1];
        fiz += fr * e[2];
    }
    __syncwarp();
    if (M.ng3eta[ei] == 0 || M.g3fast[ei]) {
        if (M.ng3eta[ei]) acsf_g3_vjp_fast<R>(M, C, ei, cnt, c, fix, fiy, fiz);
        __syncwarp();
        fix = warp_sum(fix);
        fiy = warp_sum(fiy);
        fiz = warp_sum(fiz);
        return;
    }
    const G3List g3 = g3_list(M, ei);
    TriWalk tw;
    tw.init(cnt, lane);
    while (tw.valid) {
        Triplet<R> T;
        if (triplet_setup<R>(M, C, ei, tw.q3, tw.q4, ck, T)) {
            const int ej = C.nbelem[tw.q3], ek = C.nbelem[tw.q4];
            R A1 = R(0), A2 = R(0), A3 = R(0);
            for (int u = 0; u < g3.n; ++u) {
                const int s = g3.idx[u], k = sfb + s;
                if (!g3_match(M, k, ej, ek)) continue;
                R plam, fgn;
                if (!g3_term<R>(M, k, T, plam, fgn)) continue;
                const R us = c[s] * fgn;
                A1 += us * (R)(M.zeta[k] * M.lam[k]);
                A2 += us * sf_eta<R>(M, k) * plam;
                A3 += us * plam;
            }
            const R rij = T.a[3], rik = T.c[3];
            const R P1 = T.pfc * (T.rinv0 - T.cost0 / (rij * rij)) * A1 - R(2) * T.pfc * A2 +
                         T.c[4] * T.fcjk * T.a[5] / rij * A3;
            const R P2 = T.pfc * (T.rinv0 - T.cost0 / (rik * rik)) * A1 - R(2) * T.pfc * A2 +
                         T.a[4] * T.fcjk * T.c[5] / rik * A3;
            const R P3 = T.pfc * T.rinv0 * A1 + R(2) * T.pfc * A2 - T.a[4] * T.c[4] * T.dfcjk / T.rjk * A3;
            // dxij = -a, dxik = -c, dxjk = a - c (atomsymfunction3Andi.f90:225-244):
            // F_i -= dxij P1 + dxik P2 ; F_j -= -dxij P1 - dxjk P3 ; F_k -= -dxik P2 + dxjk P3
            fix += T.a[0] * P1 + T.c[0] * P2;
            fiy += T.a[1] * P1 + T.c[1] * P2;
            fiz += T.a[2] * P1 + T.c[2] * P2;
            atomicAdd(&C.slotf[3 * tw.q3], -T.a[0] * P1 + T.jx * P3);
            atomicAdd(&C.slotf[3 * tw.q3 + 1], -T.a[1] * P1 + T.jy * P3);
            atomicAdd(&C.slotf[3 * tw.q3 + 2], -T.a[2] * P1 + T.jz * P3);
            atomicAdd(&C.slotf[3 * tw.q4], -T.c[0] * P2 - T.jx * P3);
            atomicAdd(&C.slotf[3 * tw.q4 + 1], -T.c[1] * P2 - T.jy * P3);
            atomicAdd(&C.slotf[3 * tw.q4 + 2], -T.c[2] * P2 - T.jz * P3);
        }
        tw.next();
    }
    __syncwarp();
    fix = warp_sum(fix);
    fiy = warp_sum(fiy);
    fiz = warp_sum(fiz);
}

// ---- JVP: v_s = sum_k u_k . (-dG_s/dx_k); lane 0 writes v[s] -------------------------
template <typename R>
__device__ void acsf_jvp(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, int i, const R *ux, const R *uy,
                         const R *uz, R *v) {
    const int lane = threadIdx.x & 31;
    const CutK<R> ck = cut_k<R>(M, ei);
    const R rc = ck.rc;
    const int nsf = M.nsf[ei], sfb = ei * M.maxsf;
    const R uix = ux[i], uiy = uy[i], uiz = uz[i];
    // G2: -dG/dx_i = (d/r) T', -dG/dx_j = -(d/r) T'  ->  v += T'/r d.(u_i - u_j)
    for (int s = 0; s < nsf; ++s) {
        if (M.sftype[sfb + s] != 2) continue;
        const R eta = sf_eta<R>(M, sfb + s), rs = sf_rs<R>(M, sfb + s);
        const int e1 = M.e1[sfb + s];
        R acc = R(0);
        for (int q = lane; q < cnt; q += 32) {
            const R *e = C.nb + q * C.st;
            if (C.nbelem[q] != e1 || !(e[3] <= rc)) continue;
            const int j = C.nbatom[q];
            const R ex = NM<R>::ex(-eta * (e[3] - rs) * (e[3] - rs));
            const R dt = R(-2) * eta * (e[3] - rs) * ex * e[4] + ex * e[5];
            acc += dt / e[3] * (e[0] * (uix - ux[j]) + e[1] * (uiy - uy[j]) + e[2] * (uiz - uz[j]));
        }
        acc = warp_sum(acc);
        if (lane == 0) v[s] = acc;
    }
    if (M.ng3eta[ei] == 0) {
        __syncwarp();
        return;
    }
    if (M.g3fast[ei]) {
        acsf_g3_jvp_fast<R>(M, C, ei, cnt, i, ux, uy, uz, v);
        return;
    }
    const G3List g3 = g3_list(M, ei);
    R acc[kMaxG3];
#pragma unroll
    for (int u = 0; u < kMaxG3; ++u) acc[u] = R(0);
    TriWalk tw;
    tw.init(cnt, lane);
    while (tw.valid) {
        Triplet<R> T;
        if (triplet_setup<R>(M, C, ei, tw.q3, tw.q4, ck, T)) {
            const int ej = C.nbelem[tw.q3], ek = C.nbelem[tw.q4];
            const int j = C.nbatom[tw.q3], kk = C.nbatom[tw.q4];
            // q1 = dxij.(u_i-u_j), q2 = dxik.(u_i-u_k), q3 = dxjk.(u_k-u_j)
            const R q1 = -(T.a[0] * (uix - ux[j]) + T.a[1] * (uiy - uy[j]) + T.a[2] * (uiz - uz[j]));
            const R q2 = -(T.c[0] * (uix - ux[kk]) + T.c[1] * (uiy - uy[kk]) + T.c[2] * (uiz - uz[kk]));
            const R q3 = T.jx * (ux[kk] - ux[j]) + T.jy * (uy[kk] - uy[j]) + T.jz * (uz[kk] - uz[j]);
            const R rij = T.a[3], rik = T.c[3];
            const R b1 = T.pfc * (T.rinv0 - T.cost0 / (rij * rij)), b2 = T.pfc * (T.rinv0 - T.cost0 / (rik * rik));
            const R d1 = T.c[4] * T.fcjk * T.a[5] / rij, d2 = T.a[4] * T.fcjk * T.c[5] / rik;
            const R d3 = T.a[4] * T.c[4] * T.dfcjk / T.rjk;
#pragma unroll
            for (int u = 0; u < kMaxG3; ++u) {
                if (u >= g3.n) break;
                const int k = sfb + g3.idx[u];
                if (!g3_match(M, k, ej, ek)) continue;
                R plam, fgn;
                if (!g3_term<R>(M, k, T, plam, fgn)) continue;
                const R zl = (R)(M.zeta[k] * M.lam[k]), e2 = R(2) * sf_eta<R>(M, k) * plam * T.pfc;
                const R p1 = fgn * (b1 * zl - e2 + d1 * plam);
                const R p2 = fgn * (b2 * zl - e2 + d2 * plam);
                const R p3 = fgn * (T.pfc * T.rinv0 * zl + e2 - d3 * plam);
                acc[u] -= p1 * q1 + p2 * q2 + p3 * q3;
            }
        }
        tw.next();
    }
#pragma unroll
    for (int u = 0; u < kMaxG3; ++u) {
        if (u >= g3.n) break;
        const R val = warp_sum(acc[u]);
        if (lane == 0) v[g3.idx[u]] = val;
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------
// Grid form of the G3 functions (NNDev::g3fast): cells (eta slot m, (lambda, zeta)
// slot q) share one neighbour pair; per triplet the ng exponentials and nlz angular
// powers meet in an outer product accumulated in registers.
//
// Each walk in three forms, by the set's structure (g3_form).  Most sets are a product of at most two lambdas and
// four zetas (each zeta with lambda -1 and +1): the product walk takes the powers of both p = 1 + lambda cos by one
// decoding of an exponent, in registers; compiled for 3 etas x 3 zetas and for 4 x 4, whose sums take
// registers most networks do not need (compiled for 4 x 4 alone 18.3 instead of 15.7 ms below).  Any other set of
// up to 8 cells walks its cells one by one.  512 H/graphene configurations, FP32, zeta 1, 2, 4: 4.9 ms with
// the product walk, 6.8 cell by cell; 2048 with the tensor-core network 15.7 against 20.0 ms (zeta 1, 4, 16
// fixed at compile time: 13.9); 64 in FP64 8.4 against 9.0.
// ---------------------------------------------------------------------------
constexpr int kGM = 4, kGQ = 8;  // largest grid

__device__ __forceinline__ bool fast_pair(const NNDev &M, int ei, int ej, int ek) {
    const int p1 = M.g3pair[ei][0], p2 = M.g3pair[ei][1];
    return (p1 == ej && p2 == ek) || (p2 == ej && p1 == ek);
}

// geometry of a triplet without the per-eta exponentials (computed by the caller)
template <typename R>
__device__ __forceinline__ bool triplet_geom(const NNDev &M, const WarpCache<R> &C, int q3, int q4,
                                             const CutK<R> &ck, Triplet<R> &T) {
    const R rc = ck.rc;
    T.a = C.nb + q3 * C.st;
    T.c = C.nb + q4 * C.st;
    if (!(T.a[3] <= rc && T.c[3] <= rc)) return false;
    T.jx = T.a[0] - T.c[0];
    T.jy = T.a[1] - T.c[1];
    T.jz = T.a[2] - T.c[2];
    T.rjk2 = T.jx * T.jx + T.jy * T.jy + T.jz * T.jz;
    if (!(T.rjk2 <= rc * rc)) return false;
    if constexpr (sizeof(R) == 8) {
        T.rjk = dist_of(T.rjk2, T.ijk);
    } else {
        T.rjk = NM<R>::sq(T.rjk2);
    }
    cutoff_fn<R>(M, ck, T.rjk, T.fcjk, T.dfcjk);
    T.rinv0 = NM<R>::rc(T.a[3] * T.c[3]);
    T.cost0 = (T.a[0] * T.c[0] + T.a[1] * T.c[1] + T.a[2] * T.c[2]) * T.rinv0;
    T.pfc = T.a[4] * T.c[4] * T.fcjk;
    return true;
}

// p = 1 + lambda cos with its squares p^2 .. p^16 (as far as `bits`, all exponents' bits, go), from which every
// integer power up to 31 is a product
template <typename R> struct Powers {
    R w[5];
    bool on;  // p > 0: the cells of this lambda count
    __device__ __forceinline__ Powers(R lam, R cost, int bits) {
        w[0] = R(1) + lam * cost;
        on = w[0] > R(0);
#pragma unroll
        for (int b = 1; b < 5; ++b) {
            w[b] = R(0);
            if (bits >> b) w[b] = w[b - 1] * w[b - 1];
        }
    }
};

// Any cells.  each(cos, f) calls f(q, p^(zeta-1), p^zeta) for every cell q, with zeros where p <= 0.
template <typename R> struct AnyCells {
    static constexpr int NQ = kGQ;
    R zl[NQ], lams[2];
    int zm1[NQ], bits;
    unsigned of[2];  // the cells of each of the two lambdas
    static __device__ __forceinline__ int sf(const NNDev &M, int ei, int m, int q) {
        return q < M.nlz[ei] ? M.sf_of[ei][m][q] : -1;
    }
    static __device__ __forceinline__ R pn(const NNDev &M, int ei, int q) {
        return q < M.nlz[ei] ? widen<R>(M.lz_pnorm[ei][q]) : R(0);
    }
    __device__ __forceinline__ AnyCells(const NNDev &M, int ei) {
        bits = 0;
        lams[0] = widen<R>(M.lz_lam[ei][0]);
        lams[1] = R(0);
        of[0] = of[1] = 0u;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            zl[q] = R(0);
            zm1[q] = 0;
            if (q >= M.nlz[ei]) continue;
            zl[q] = widen<R>(M.lz_zl[ei][q]);
            zm1[q] = M.lz_zm1[ei][q];
            bits |= zm1[q];
            if (M.lz_lam[ei][q] == M.lz_lam[ei][0]) {
                of[0] |= 1u << q;
            } else {
                lams[1] = widen<R>(M.lz_lam[ei][q]);
                of[1] |= 1u << q;
            }
        }
    }
    template <typename F> __device__ __forceinline__ void each(R cost, F f) const {
#pragma unroll
        for (int l = 0; l < 2; ++l) {
            if (!of[l]) continue;
            const Powers<R> L(lams[l], cost, bits);
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                if (!(of[l] >> q & 1u)) continue;
                R r = zm1[q] & 1 ? L.w[0] : R(1);
#pragma unroll
                for (int b = 1; b < 5; ++b)
                    if ((zm1[q] >> b) & 1) r *= L.w[b];
                f(q, L.on ? r : R(0), L.on ? r * L.w[0] : R(0));
            }
        }
    }
};

// the product of two lambdas and NZ zetas, cell 2 z + l (cells that are not in the set have no function)
template <typename R, int NZ> struct ProductCells {
    static constexpr int NQ = 2 * NZ;
    R zl[NQ], lams[2];
    int ex[NZ], bits;
    static __device__ __forceinline__ int sf(const NNDev &M, int ei, int m, int q) { return M.gsf[ei][m][q]; }
    static __device__ __forceinline__ R pn(const NNDev &M, int ei, int q) { return widen<R>(M.gpn[ei][q >> 1]); }
    __device__ __forceinline__ ProductCells(const NNDev &M, int ei) {
        bits = 0;
#pragma unroll
        for (int l = 0; l < 2; ++l) lams[l] = widen<R>(M.glam[ei][l]);
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
            ex[z] = M.gex[ei][z];
            bits |= ex[z];
#pragma unroll
            for (int l = 0; l < 2; ++l) zl[2 * z + l] = widen<R>((float)(ex[z] + 1) * M.glam[ei][l]);
        }
    }
    template <typename F> __device__ __forceinline__ void each(R cost, F f) const {
        const Powers<R> L0(lams[0], cost, bits), L1(lams[1], cost, bits);
#pragma unroll
        for (int z = 0; z < NZ; ++z) {
            R r0 = R(1), r1 = R(1);
            if (ex[z] & 1) {
                r0 = L0.w[0];
                r1 = L1.w[0];
            }
#pragma unroll
            for (int b = 1; b < 5; ++b)
                if ((ex[z] >> b) & 1) {
                    r0 *= L0.w[b];
                    r1 *= L1.w[b];
                }
            f(2 * z, L0.on ? r0 : R(0), L0.on ? r0 * L0.w[0] : R(0));
            f(2 * z + 1, L1.on ? r1 : R(0), L1.on ? r1 * L1.w[0] : R(0));
        }
    }
};

// exp(-eta_m (r_ij^2 + r_ik^2 + r_jk^2)) for every eta slot
template <typename R, int GM>
__device__ __forceinline__ void grid_pexp(const R *eta, int ng, const Triplet<R> &T, R *E) {
#pragma unroll
    for (int m = 0; m < GM; ++m) E[m] = m < ng ? T.a[6 + m] * T.c[6 + m] * NM<R>::ex(-eta[m] * T.rjk2) : R(0);
}

// forces of one triplet from its A1, A2, A3 (head of this file): on the centre, the row's neighbour
// and the neighbour q4
template <typename R>
__device__ __forceinline__ void vjp_pairs(const Triplet<R> &T, R A1, R A2, R A3, const WarpCache<R> &C, int q4, R &fix,
                                          R &fiy, R &fiz, R &sjx, R &sjy, R &sjz) {
    const R rij = T.a[3], rik = T.c[3];
    R P1, P2, P3;
    if constexpr (sizeof(R) == 8) {
        // 1/r_ij = r_ik/(r_ij r_ik) and so on: products for the five divisions
        const R iij = T.rinv0 * rik, iik = T.rinv0 * rij, ijk = T.ijk, w = R(2) * T.pfc * A2;
        P1 = T.pfc * (T.rinv0 - T.cost0 * (iij * iij)) * A1 - w + T.c[4] * T.fcjk * T.a[5] * iij * A3;
        P2 = T.pfc * (T.rinv0 - T.cost0 * (iik * iik)) * A1 - w + T.a[4] * T.fcjk * T.c[5] * iik * A3;
        P3 = T.pfc * T.rinv0 * A1 + w - T.a[4] * T.c[4] * T.dfcjk * ijk * A3;
    } else {
        P1 = T.pfc * (T.rinv0 - T.cost0 / (rij * rij)) * A1 - R(2) * T.pfc * A2 +
             T.c[4] * T.fcjk * T.a[5] / rij * A3;
        P2 = T.pfc * (T.rinv0 - T.cost0 / (rik * rik)) * A1 - R(2) * T.pfc * A2 +
             T.a[4] * T.fcjk * T.c[5] / rik * A3;
        P3 = T.pfc * T.rinv0 * A1 + R(2) * T.pfc * A2 - T.a[4] * T.c[4] * T.dfcjk / T.rjk * A3;
    }
    fix += T.a[0] * P1 + T.c[0] * P2;
    fiy += T.a[1] * P1 + T.c[1] * P2;
    fiz += T.a[2] * P1 + T.c[2] * P2;
    sjx += -T.a[0] * P1 + T.jx * P3;
    sjy += -T.a[1] * P1 + T.jy * P3;
    sjz += -T.a[2] * P1 + T.jz * P3;
    atomicAdd(&C.slotf[3 * q4], -T.c[0] * P2 - T.jx * P3);
    atomicAdd(&C.slotf[3 * q4 + 1], -T.c[1] * P2 - T.jy * P3);
    atomicAdd(&C.slotf[3 * q4 + 2], -T.c[2] * P2 - T.jz * P3);
}

template <typename R, int GM, typename CELLS>
__device__ __forceinline__ void g3_forward_walk(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, R *G) {
    const int lane = threadIdx.x & 31, ng = M.ng3eta[ei];
    constexpr int GQ = CELLS::NQ;
    const CutK<R> ck = cut_k<R>(M, ei);
    const CELLS g(M, ei);
    R eta[GM];
#pragma unroll
    for (int m = 0; m < GM; ++m) eta[m] = m < ng ? g3_eta<R>(M, ei, m) : R(0);
    R acc[GM][GQ];
#pragma unroll
    for (int m = 0; m < GM; ++m)
#pragma unroll
        for (int q = 0; q < GQ; ++q) acc[m][q] = R(0);
    RowWalk tw;
    tw.init(cnt, lane);
    while (tw.valid) {
        Triplet<R> T;
        if (fast_pair(M, ei, C.nbelem[tw.q3], C.nbelem[tw.q4]) && triplet_geom<R>(M, C, tw.q3, tw.q4, ck, T)) {
            R E[GM];
            grid_pexp<R, GM>(eta, ng, T, E);
#pragma unroll
            for (int m = 0; m < GM; ++m) E[m] *= T.pfc;
            g.each(T.cost0, [&](int q, R, R pw) {
#pragma unroll
                for (int m = 0; m < GM; ++m) acc[m][q] += E[m] * pw;
            });
        }
        tw.next();
    }
#pragma unroll
    for (int m = 0; m < GM; ++m)
#pragma unroll
        for (int q = 0; q < GQ; ++q) {
            const int s = m < ng ? CELLS::sf(M, ei, m, q) : -1;
            if (s < 0) continue;
            const R v = warp_sum(acc[m][q]);
            if (lane == 0) G[s] = v * CELLS::pn(M, ei, q);
        }
    __syncwarp();
}

// G3 part of the VJP in grid form; adds into fix/fiy/fiz and the slot forces
template <typename R, int GM, typename CELLS>
__device__ __forceinline__ void g3_vjp_walk(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, const R *c, R &fix,
                                            R &fiy, R &fiz) {
    const int lane = threadIdx.x & 31, ng = M.ng3eta[ei];
    constexpr int GQ = CELLS::NQ;
    const CutK<R> ck = cut_k<R>(M, ei);
    const CELLS g(M, ei);
    R eta[GM];
#pragma unroll
    for (int m = 0; m < GM; ++m) eta[m] = m < ng ? g3_eta<R>(M, ei, m) : R(0);
    R Wc[GM][GQ];
#pragma unroll
    for (int m = 0; m < GM; ++m)
#pragma unroll
        for (int q = 0; q < GQ; ++q) {
            const int s = m < ng ? CELLS::sf(M, ei, m, q) : -1;
            Wc[m][q] = s >= 0 ? c[s] * CELLS::pn(M, ei, q) : R(0);
        }
    R sjx = R(0), sjy = R(0), sjz = R(0);  // force on the current row's neighbour q3
    RowWalk tw;
    tw.init(cnt, lane);
    while (tw.valid) {
        Triplet<R> T;
        if (fast_pair(M, ei, C.nbelem[tw.q3], C.nbelem[tw.q4]) && triplet_geom<R>(M, C, tw.q3, tw.q4, ck, T)) {
            R E[GM];
            grid_pexp<R, GM>(eta, ng, T, E);
            R A1 = R(0), A2 = R(0), A3 = R(0);
            g.each(T.cost0, [&](int q, R pp, R pl) {
                R S = R(0), Tq = R(0);
#pragma unroll
                for (int m = 0; m < GM; ++m) {
                    const R w = Wc[m][q] * E[m];
                    S += w;
                    Tq += eta[m] * w;
                }
                A1 += g.zl[q] * pp * S;
                A2 += pl * Tq;
                A3 += pl * S;
            });
            vjp_pairs<R>(T, A1, A2, A3, C, tw.q4, fix, fiy, fiz, sjx, sjy, sjz);
        }
        if (tw.row_end) {
            atomicAdd(&C.slotf[3 * tw.q3], sjx);
            atomicAdd(&C.slotf[3 * tw.q3 + 1], sjy);
            atomicAdd(&C.slotf[3 * tw.q3 + 2], sjz);
            sjx = sjy = sjz = R(0);
        }
        tw.next();
    }
}

// G3 part of the JVP in grid form; lane 0 writes v[s]
template <typename R, int GM, typename CELLS>
__device__ __forceinline__ void g3_jvp_walk(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, int i, const R *ux,
                                            const R *uy, const R *uz, R *v) {
    const int lane = threadIdx.x & 31, ng = M.ng3eta[ei];
    constexpr int GQ = CELLS::NQ;
    const CutK<R> ck = cut_k<R>(M, ei);
    const CELLS g(M, ei);
    R eta[GM];
#pragma unroll
    for (int m = 0; m < GM; ++m) eta[m] = m < ng ? g3_eta<R>(M, ei, m) : R(0);
    const R uix = ux[i], uiy = uy[i], uiz = uz[i];
    R acc[GM][GQ];
#pragma unroll
    for (int m = 0; m < GM; ++m)
#pragma unroll
        for (int q = 0; q < GQ; ++q) acc[m][q] = R(0);
    RowWalk tw;
    tw.init(cnt, lane);
    while (tw.valid) {
        Triplet<R> T;
        if (fast_pair(M, ei, C.nbelem[tw.q3], C.nbelem[tw.q4]) && triplet_geom<R>(M, C, tw.q3, tw.q4, ck, T)) {
            const int j = C.nbatom[tw.q3], kk = C.nbatom[tw.q4];
            const R q1 = -(T.a[0] * (uix - ux[j]) + T.a[1] * (uiy - uy[j]) + T.a[2] * (uiz - uz[j]));
            const R q2 = -(T.c[0] * (uix - ux[kk]) + T.c[1] * (uiy - uy[kk]) + T.c[2] * (uiz - uz[kk]));
            const R q3 = T.jx * (ux[kk] - ux[j]) + T.jy * (uy[kk] - uy[j]) + T.jz * (uz[kk] - uz[j]);
            const R rij = T.a[3], rik = T.c[3];
            const R b1 = T.pfc * (T.rinv0 - T.cost0 / (rij * rij)), b2 = T.pfc * (T.rinv0 - T.cost0 / (rik * rik));
            const R d1 = T.c[4] * T.fcjk * T.a[5] / rij, d2 = T.a[4] * T.fcjk * T.c[5] / rik;
            const R d3 = T.a[4] * T.c[4] * T.dfcjk / T.rjk;
            const R X1 = b1 * q1 + b2 * q2 + T.pfc * T.rinv0 * q3, X2 = T.pfc * (q1 + q2 - q3),
                    X3 = d1 * q1 + d2 * q2 - d3 * q3;
            R E[GM];
            grid_pexp<R, GM>(eta, ng, T, E);
            g.each(T.cost0, [&](int q, R pp, R pl) {
                const R t1 = g.zl[q] * X1, t2 = R(2) * X2;
#pragma unroll
                for (int m = 0; m < GM; ++m) acc[m][q] -= E[m] * (pp * t1 + pl * (X3 - eta[m] * t2));
            });
        }
        tw.next();
    }
#pragma unroll
    for (int m = 0; m < GM; ++m)
#pragma unroll
        for (int q = 0; q < GQ; ++q) {
            const int s = m < ng ? CELLS::sf(M, ei, m, q) : -1;
            if (s < 0) continue;
            const R val = warp_sum(acc[m][q]);
            if (lane == 0) v[s] = val * CELLS::pn(M, ei, q);
        }
    __syncwarp();
}

// calls f(GM, cells) of the form of element ei's walk
template <typename R, typename F> __device__ __forceinline__ void g3_form(const NNDev &M, int ei, F f) {
    const int nz = M.gz[ei];
    if (nz == 0) f(std::integral_constant<int, kGM>(), (AnyCells<R> *)nullptr);
    else if (nz <= 3 && M.ng3eta[ei] <= 3) f(std::integral_constant<int, 3>(), (ProductCells<R, 3> *)nullptr);
    else f(std::integral_constant<int, 4>(), (ProductCells<R, 4> *)nullptr);
}

template <typename R> __device__ void acsf_g3_forward_fast(const NNDev &M, const WarpCache<R> &C, int ei, int cnt,
                                                           R *G) {
    g3_form<R>(M, ei, [&](auto gm, auto *cells) {
        g3_forward_walk<R, decltype(gm)::value, std::remove_reference_t<decltype(*cells)>>(M, C, ei, cnt, G);
    });
}

template <typename R>
__device__ void acsf_g3_vjp_fast(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, const R *c, R &fix, R &fiy,
                                 R &fiz) {
    g3_form<R>(M, ei, [&](auto gm, auto *cells) {
        g3_vjp_walk<R, decltype(gm)::value, std::remove_reference_t<decltype(*cells)>>(M, C, ei, cnt, c, fix, fiy, fiz);
    });
}

template <typename R>
__device__ void acsf_g3_jvp_fast(const NNDev &M, const WarpCache<R> &C, int ei, int cnt, int i, const R *ux,
                                 const R *uy, const R *uz, R *v) {
    g3_form<R>(M, ei, [&](auto gm, auto *cells) {
        g3_jvp_walk<R, decltype(gm)::value, std::remove_reference_t<decltype(*cells)>>(M, C, ei, cnt, i, ux, uy, uz, v);
    });
}

}  // namespace mdt
