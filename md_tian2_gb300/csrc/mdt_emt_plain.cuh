// mdt_emt_plain.cuh -- EMT of one bead with FP64 forces in its short form: one walk over all pairs,
// both ends added to shared memory.  The FP32 network kernels' fallback for a trajectory whose
// descriptors left the training range (a few in a million bead evaluations).  emt_beads
// (mdt_emt.cuh) is 1.6 times faster, but inlined next to the walks of those kernels, which hold
// all 128 registers a thread may have, it costs spills there: 79 -> 83 ms for 100 steps of the
// 4096-trajectory surrogate batch (as a call 88 ms), 76-77 ms with this form.
//
// Pair layout: pair (i, j = (i+k) mod N), k = 1..N/2, in scratch slot (k-1) N + i (the k = N/2
// row holds only i < N/2 when N is even): d, Q_ij, Q_ji and the pair-potential scalar F_V.
#pragma once
#include "mdt_emt.cuh"

namespace mdt {

// Adds forces into B.f*, sets dens, adds the bead's energy into B.epot.  Must be called by all
// threads of the CTA.
static __device__ void emt_bead_plain(const Batch &B, const EmtConst &E, const SmemEmt<double> &S, int t, int b,
                         bool do_forces) {
    using R = double;
    int8_t *const s_typ = (int8_t *)S.perm, *const s_slot = s_typ + B.max_atoms;
    const int N = B.natoms[t];
    const int64_t base = B.ba_off[t] + (int64_t)b * N;
    const int aoff = B.atom_off[t];
    const int tid = threadIdx.x, nt = blockDim.x;

    for (int i = tid; i < N; i += nt) {
        S.px[i] = B.rx[base + i];
        S.py[i] = B.ry[base + i];
        S.pz[i] = B.rz[base + i];
        const int ty = B.type[aoff + i];
        s_typ[i] = (int8_t)ty;
        s_slot[i] = (int8_t)E.slot_of_type[ty];
        S.sig[i] = R(0);
        S.fx[i] = R(0);
        S.fy[i] = R(0);
        S.fz[i] = R(0);
    }
    load_cell(B, t, *S.cell);
    __syncthreads();
    const Cell &cell = *S.cell;

    const int K = N / 2, NK = N * K;
    R *scr = (R *)B.pair_scratch + 6 * (B.pair_off[t] + (int64_t)b * NK);
    R *s_dx = scr, *s_dy = scr + NK, *s_dz = scr + 2 * NK, *s_qij = scr + 3 * NK, *s_qji = scr + 4 * NK,
      *s_fv = scr + 5 * NK;
    const R cut2 = (R)E.cut2, acut = (R)E.acut, rcut = (R)E.rcut;
    double e_pair = 0.0;

    // ---- pass 1 (pair-parallel; consecutive threads take consecutive atoms i of one
    // k row, so their shared-memory atomics hit distinct atoms) --------------------
    for (int p = tid; p < NK; p += nt) {
        const int k = p / N + 1, i = p - (k - 1) * N;
        int j = i + k;
        if (j >= N) j -= N;
        const int ti = s_typ[i], tj = s_typ[j];
        R q_ij = R(0), q_ji = R(0), fv = R(0), rx = R(0), ry = R(0), rz = R(0);
        if (!(2 * k == N && i >= K) && ((E.pair_mask >> (ti * kMaxTypes + tj)) & 1u)) {
            min_image(cell, S.px[i] - S.px[j], S.py[i] - S.py[j], S.pz[i] - S.pz[j], rx, ry, rz);
            const R r2 = rx * rx + ry * ry + rz * rz;
            // skipped only beyond the cutoff, like the reference's `if (r > cutoff*rcut) cycle`
            // (pes_emt_mod.f90:660): a distance that is not a number enters the sums
            if (!(r2 > cut2)) {
                const R ir = Math<R>::rsq(r2), r = r2 * ir;
                const R e = Math<R>::ex(acut * (r - rcut));
                const R theta = Math<R>::rcp(R(1) + e);
                const R rt1 = acut * e * theta;
                const int si = s_slot[i], sj = s_slot[j];
                const R phi_j = theta * Math<R>::ex(-(R)E.eta2[sj] * (r - (R)E.betas0[sj]));
                const R psi_j = theta * Math<R>::ex(-(R)E.kappadbeta[sj] * (r - (R)E.betas0[sj]));
                R phi_i = phi_j, psi_i = psi_j;
                if (si != sj) {
                    phi_i = theta * Math<R>::ex(-(R)E.eta2[si] * (r - (R)E.betas0[si]));
                    psi_i = theta * Math<R>::ex(-(R)E.kappadbeta[si] * (r - (R)E.betas0[si]));
                }
                const R gij = (R)(E.igamma1[si] * E.chi[si][sj]);
                const R gji = (R)(E.igamma1[sj] * E.chi[sj][si]);
                atomicAdd(&S.sig[i], gij * phi_j);
                atomicAdd(&S.sig[j], gji * phi_i);
                const R cij = (R)(E.g2v0[si] * E.chi[si][sj]);
                const R cji = (R)(E.g2v0[sj] * E.chi[sj][si]);
                e_pair -= 0.5 * (double)(cij * psi_j + cji * psi_i);
                fv = -R(0.5) * (cij * ((R)E.kappadbeta[sj] + rt1) * psi_j +
                                cji * ((R)E.kappadbeta[si] + rt1) * psi_i) * ir;
                R eta_j = (R)E.eta2[sj], eta_i = (R)E.eta2[si];
                // QUIRK kept from pes_emt_mod.f90:705: the type1-type1 density
                // derivative uses eta2 of type2.
                if (E.hh_quirk && si == 0 && sj == 0) eta_j = eta_i = (R)E.eta2[1];
                q_ij = gij * (eta_j + rt1) * phi_j * ir;
                q_ji = gji * (eta_i + rt1) * phi_i * ir;
            }
        }
        if (do_forces) {
            s_dx[p] = rx;
            s_dy[p] = ry;
            s_dz[p] = rz;
            s_qij[p] = q_ij;
            s_qji[p] = q_ji;
            s_fv[p] = fv;
        }
    }
    __syncthreads();

    // ---- per-atom epilogue ---------------------------------------------------
    double e_atom = 0.0;
    for (int i = tid; i < N; i += nt) {
        const int s = s_slot[i];
        if (s < 0) {
            S.A[i] = R(0);
            continue;
        }
        const double sc = fmax((double)1e-30f, (double)S.sig[i]);  // single-precision 1e-30, pes_emt_mod.f90:793
        const double sa = -log(fmax(kTolerance, sc) * kTwelfth) / E.betaeta2[s];
        const double el = exp_t64(-E.lambda[s] * sa), ek = exp_t64(-E.kappa[s] * sa);
        e_atom += E.e0[s] * ((1.0 + E.lambda[s] * sa) * el - 1.0) + 6.0 * E.v0[s] * ek;
        const double W = E.e0[s] * E.lambda[s] * E.lambda[s] * sa * el + 6.0 * E.v0[s] * E.kappa[s] * ek;
        S.A[i] = (R)(W / (E.betaeta2[s] * sc));
        B.dens[base + i] = E.n0[s] * exp_t64(E.dens_exp[s] * sa);
    }
    const double etot = block_sum(e_pair + e_atom, S.red);  // contains __syncthreads
    if (tid == 0) B.epot[B.bead_off[t] + b] += etot;
    if (!do_forces) return;

    // ---- pass 2 (gather): work item (i, chunk of k); consecutive threads take
    // consecutive atoms, partial forces meet in shared memory ----------------------
    const int C = (N >= nt) ? 1 : min(K > 0 ? K : 1, nt / N);
    const int per = (K + C - 1) / C;
    for (int w = tid; w < N * C; w += nt) {
        const int c = w / N, i = w - c * N;
        const int k0 = 1 + c * per, k1 = min(K, (c + 1) * per);
        const R Ai = S.A[i];
        R fx = R(0), fy = R(0), fz = R(0);
        for (int k = k0; k <= k1; ++k) {
            const bool half = (2 * k == N);
            int j = i + k;
            if (j >= N) j -= N;
            if (!(half && i >= K)) {  // i is the first atom of pair (i, i+k)
                const int p = (k - 1) * N + i;
                const R cc = Ai * s_qij[p] + S.A[j] * s_qji[p] + s_fv[p];
                fx += cc * s_dx[p];
                fy += cc * s_dy[p];
                fz += cc * s_dz[p];
            }
            int m = i - k;
            if (m < 0) m += N;
            if (!(half && m >= K)) {  // i is the second atom of pair (m, m+k)
                const int p = (k - 1) * N + m;
                const R cc = S.A[m] * s_qij[p] + Ai * s_qji[p] + s_fv[p];
                fx -= cc * s_dx[p];
                fy -= cc * s_dy[p];
                fz -= cc * s_dz[p];
            }
        }
        if (C == 1) {
            S.fx[i] = fx;
            S.fy[i] = fy;
            S.fz[i] = fz;
        } else {
            atomicAdd(&S.fx[i], fx);
            atomicAdd(&S.fy[i], fy);
            atomicAdd(&S.fz[i], fz);
        }
    }
    __syncthreads();
    for (int i = tid; i < N; i += nt) {
        B.fx[base + i] += (double)S.fx[i];
        B.fy[base + i] += (double)S.fy[i];
        B.fz[base + i] += (double)S.fz[i];
    }
    __syncthreads();
}

}  // namespace mdt
