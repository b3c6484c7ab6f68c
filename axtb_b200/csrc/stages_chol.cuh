// Cholesky factor and triangular inverse of the staged molecules' overlap matrices (and EEQ matrices),
// the same blocks of 64 as team_cholesky and team_trinv, a launch per step over molecules of like size
// (cholesky_plan):
//   k_ch_init    the matrix into place; the first diagonal block factored and inverted
//   k_ch_panel   step p: L[i, p] = A[i, p] L[p, p]^-T below, and row block p of the inverse,
//                X[p, j] = -L[p, p]^-1 (L[p, j:p] X[j:p, j]), a 64 x 64 tile per CTA
//   k_ch_trail   step p: A[i, j] -= L[i, p] L[j, p]^T, and the next diagonal block factored and
//                inverted by the CTA that has just updated it
// (crates/base/src/linalg/eigen.rs:72-113, crates/axtb/src/eeq.rs:43-77). One CTA took a molecule's
// blocks one after the other before, with the factor and its inverse in two passes of ~25 and ~40 us
// per block; the two now share their 64 steps (one column of L and one row of the inverse each).
#pragma once
#include "stages.cuh"

namespace axg {

// The matrices of a molecule: the overlap (factor in scr1, inverse in Linv) or the EEQ matrix
struct ChSystem {
    int n;
    double *L, *X, *bad;  // bad: nonzero when a pivot was not positive
};
__device__ __forceinline__ ChSystem ch_system(const Batch& B, const State& S, const TeamPlan& P, int m, int eeq) {
    double* wk = P.wk + P.m_wk0[m];
    if (eeq) return {B.m_nat[m], S.eeq_A + P.m_sq0[m], S.eeq_A + P.eeq_plane + P.m_sq0[m], wk + 1};
    return {B.m_nao[m], S.scr1 + B.m_mat0[m], S.Linv + B.m_mat0[m], wk + 1};
}

// Diagonal block p: L_pp and its inverse. Step j scales column j of the block and row j of the
// inverse by 1 / l_jj, then takes column j out of both (thread = a column, four rows at a time).
__device__ void ch_factor(const ChSystem& s, int p, int* status, int eeq) {
    constexpr int LP = CB + 1;
    double *a = s_work, *x = s_work + CB * LP;  // [row * LP + column]
    const int r0 = p * CB, nb = min(CB, s.n - r0), tid = threadIdx.x;
    double* A = s.L + r0 + (long long)r0 * s.n;
    __syncthreads();
    for (int e = tid; e < CB * CB; e += TEAM_THREADS) {
        int r = e % CB, c = e / CB;
        a[r * LP + c] = r < nb && c <= r ? A[r + (long long)c * s.n] : (r == c ? 1.0 : 0.0);
        x[r * LP + c] = r == c ? 1.0 : 0.0;
    }
    __syncthreads();
    bool ok = true;
    const int c = tid & 63, rw = tid >> 6;
    for (int j = 0; j < nb; j++) {
        double d = a[j * LP + j];
        if (!(d > 0.0)) {
            ok = false;
            d = 1.0;
        }
        const double l = sqrt(d), inv = 1.0 / l;
        __syncthreads();  // the pivot has been read
        if (rw == 0) {
            if (c > j) a[c * LP + j] *= inv;
            else x[j * LP + c] *= inv;
            if (c == j) a[j * LP + j] = l;
        }
        __syncthreads();
        double* t = c <= j ? x : a;
        const double f = c <= j ? x[j * LP + c] : a[c * LP + j];
        const int first = c <= j ? j + 1 : c;  // the lower triangle of a only
        for (int r = first + ((rw - first) & 3); r < nb; r += 4) t[r * LP + c] = fma(-a[r * LP + j], f, t[r * LP + c]);
        __syncthreads();
    }
    double* X = s.X + r0 + (long long)r0 * s.n;
    for (int e = tid; e < nb * nb; e += TEAM_THREADS) {
        int r = e % nb, q = e / nb;
        if (r >= q) A[r + (long long)q * s.n] = a[r * LP + q];
        X[r + (long long)q * s.n] = r >= q ? x[r * LP + q] : 0.0;
    }
    if (!ok && tid == 0) {
        *s.bad = 1.0;
        if (!eeq) atomicOr(status, ST_NOT_PD);
    }
}

// tile (blockIdx.x) of molecule Q.mol[blockIdx.y]: the overlap copied, the inverse's upper part zero
__global__ void __launch_bounds__(TEAM_THREADS, 2) k_ch_init(Batch B, State S, StagePlan Q, TeamPlan P, int eeq) {
    const int m = Q.mol[blockIdx.y];
    const ChSystem s = ch_system(B, S, P, m, eeq);
    const int rt = (s.n + CB - 1) / CB;
    if ((int)blockIdx.x >= rt * rt) return;
    const int bi = blockIdx.x % rt, bj = blockIdx.x / rt;
    if (blockIdx.x == 0 && threadIdx.x == 0) *s.bad = 0.0;
    for (int e = threadIdx.x; e < CB * CB; e += TEAM_THREADS) {
        int r = bi * CB + e % CB, c = bj * CB + e / CB;
        if (r >= s.n || c >= s.n) continue;
        const long long o = r + (long long)c * s.n;
        if (!eeq && bi >= bj) s.L[o] = S.S[B.m_mat0[m] + o];
        if (bi < bj) s.X[o] = 0.0;
    }
    if (blockIdx.x == 0) {
        __syncthreads();
        ch_factor(s, 0, &S.status[m], eeq);
    }
}

__global__ void __launch_bounds__(TEAM_THREADS, 2) k_ch_panel(Batch B, State S, StagePlan Q, TeamPlan P, int p, int eeq) {
    const int m = Q.mol[blockIdx.y];
    const ChSystem s = ch_system(B, S, P, m, eeq);
    const int n = s.n, rt = (n + CB - 1) / CB;
    if (p >= rt || (int)blockIdx.x >= rt - 1) return;
    const int nb = min(CB, n - p * CB);
    const Team t{0, 1, false};
    const double* Xpp = s.X + p * CB + (long long)p * CB * n;
    if ((int)blockIdx.x < p) {  // the inverse: longest sums first
        const int j = blockIdx.x;
        double* Xpj = s.X + p * CB + (long long)j * CB * n;
        team_gemm(t, false, false, nb, CB, (p - j) * CB, -1.0, s.L + p * CB + (long long)j * CB * n, n,
                  s.X + j * CB + (long long)j * CB * n, n, 0.0, Xpj, n);
        __syncthreads();
        // in place: the one output tile reads all of itself before its first store
        team_gemm(t, false, false, nb, CB, nb, 1.0, Xpp, n, Xpj, n, 0.0, Xpj, n);
    } else {
        const int i = blockIdx.x + 1;
        double* Aip = s.L + i * CB + (long long)p * CB * n;
        team_gemm(t, false, true, min(CB, n - i * CB), nb, nb, 1.0, Aip, n, Xpp, n, 0.0, Aip, n);
    }
}

__global__ void __launch_bounds__(TEAM_THREADS, 2) k_ch_trail(Batch B, State S, StagePlan Q, TeamPlan P, int p, int eeq) {
    const int m = Q.mol[blockIdx.y];
    const ChSystem s = ch_system(B, S, P, m, eeq);
    const int n = s.n, rt = (n + CB - 1) / CB, left = rt - 1 - p;
    if (left <= 0 || (int)blockIdx.x >= left * (left + 1) / 2) return;
    int j = 0, tile = blockIdx.x;
    while (tile >= left - j) tile -= left - j, j++;
    const int bj = p + 1 + j, bi = bj + tile;
    const double* Lp = s.L + (long long)p * CB * n;
    team_gemm(Team{0, 1, false}, false, true, min(CB, n - bi * CB), min(CB, n - bj * CB), CB, -1.0, Lp + bi * CB, n,
              Lp + bj * CB, n, 1.0, s.L + bi * CB + (long long)bj * CB * n, n);
    if (blockIdx.x == 0) {  // tile (p + 1, p + 1)
        __syncthreads();
        ch_factor(s, p + 1, &S.status[m], eeq);
    }
}

// EEQ charges from the inverse factor X of J: J^-1 b = X^T (X b) for b = the right-hand side and b = 1,
// then the charge constraint (mol_eeq). part 0: X b, 32 rows per CTA; 1: X^T (..), a warp per column;
// 2: the constraint, a CTA per molecule. The vectors wait in the molecule's workspace.
__global__ void __launch_bounds__(TEAM_THREADS) k_ch_eeq(Batch B, State S, StagePlan Q, TeamPlan P, int part) {
    const int m = Q.mol[blockIdx.y];
    const ChSystem s = ch_system(B, S, P, m, 1);
    const int n = s.n, a0 = B.m_at0[m], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *y0 = P.wk + P.m_wk0[m] + 8, *y1 = y0 + n, *z1 = y1 + n;
    if (part == 0) {
        __shared__ double p0[8][32], p1[8][32];
        const int r = 32 * blockIdx.x + lane;
        if (32 * (int)blockIdx.x >= n) return;
        double u = 0.0, v = 0.0;
        if (r < n)
            for (int c = warp; c <= r; c += 8) {
                const double x = s.X[r + (long long)c * n];
                u = fma(x, P.eeq_rhs[a0 + c], u);
                v += x;
            }
        p0[warp][lane] = u;
        p1[warp][lane] = v;
        __syncthreads();
        if (warp == 0 && r < n) {
            for (int q = 1; q < 8; q++) u += p0[q][lane], v += p1[q][lane];
            y0[r] = u;
            y1[r] = v;
        }
    } else if (part == 1) {
        const int c = 8 * blockIdx.x + warp;
        if (c >= n) return;
        double u = 0.0, v = 0.0;
        for (int r = c + lane; r < n; r += 32) {
            const double x = s.X[r + (long long)c * n];
            u = fma(x, y0[r], u);
            v = fma(x, y1[r], v);
        }
        u = warp_sum(u);
        v = warp_sum(v);
        if (lane == 0) {
            P.eeq_q[a0 + c] = u;
            z1[c] = v;
        }
    } else {
        double sa = 0.0, sb = 0.0;
        for (int i = threadIdx.x; i < n; i += TEAM_THREADS) {
            sa += P.eeq_q[a0 + i];
            sb += z1[i];
        }
        const Team t{0, 1, false};
        sa = team_sum(t, sa, nullptr);
        sb = team_sum(t, sb, nullptr);
        const double lam = (sa - B.m_charge[m]) / sb;
        for (int i = threadIdx.x; i < n; i += TEAM_THREADS) {
            double q = P.eeq_q[a0 + i] - lam * z1[i];
            if (*s.bad != 0.0 || !isfinite(q)) q = 0.0;  // neutral-atom start when the EEQ system fails
            P.eeq_q[a0 + i] = q;
        }
    }
}

}  // namespace axg
