// The eigen phase of the molecules whose tridiagonal reduction runs on chip (trd.cuh), one launch
// per stage over all of them, each stage cut into the tasks that are independent in it:
//   k_st_tiles32 32 x 32 tiles of X = L^-1 F, F' = X L^-T, C = L^-T Z, P = (C f) C^T, W
//                (k_st_tiles: 64 x 64, for split precision)
//   k_st_bisect  32 orbital energies per CTA
//   k_st_fermi   the filling, a CTA per molecule
//   k_st_invit   one eigenvector of the tridiagonal matrix per thread, 32 per CTA
//   k_st_gs      the clusters of close levels, a warp each
//   k_st_tfac    the triangular factor of 64 reflectors per CTA
//   k_st_apply   the back-transformation of a few columns per CTA, all reflectors in turn
// (crates/base/src/linalg/eigen.rs:213-296, occupations.rs:94-179, density.rs:65-87). In the team
// kernel one CTA did all of this for its molecule: a single molecule used one of 148 SMs, and a
// batch's launch was as long as its largest molecule's chain. Here a task never waits for another,
// no task's arithmetic depends on how many there are, and the molecules' bits do not depend on
// the batch.
#pragma once
#include "team_kernel.cuh"

namespace axg {

// the staged molecules and their task offsets (prefix sums over the list)
struct StagePlan {
    int count;
    const int* mol;
    const long long* off_full;   // rt^2 tiles, rt = ceil(n / 64)
    const long long* off_low;    // rt (rt + 1) / 2 tiles on and below the diagonal
    const long long* off_full32; // the same in tiles of 32
    const long long* off_low32;
    const long long* off_rt;     // rt blocks of 64
    const long long* off_vec;    // ceil(n / 32) blocks of 32 levels or vectors
    const long long* off_col;    // column blocks of the back-transformation
    const int* width;            // ... and their width (8 or 24), per molecule
};

// Profiling runs (instances of the kernels with PROF): SM cycles of a stage's CTA into its molecule's counter
// and the profiler's slot of the part (mol_eigen's slots), in units of the team kernel's half-SM CTAs (by
// threads).
template <bool PROF>
__device__ __forceinline__ long long& stage_t0() {
    __shared__ long long t0;
    return t0;
}
template <bool PROF>
__device__ __forceinline__ void stage_start() {
    if constexpr (PROF)
        if (threadIdx.x == 0) stage_t0<PROF>() = clock64();
}
template <bool PROF>
__device__ __forceinline__ void stage_stop(const State& S, int m, int slot, int thread = 0) {
    if constexpr (PROF)
        if ((int)threadIdx.x == thread) {
            const double c = (double)(clock64() - stage_t0<PROF>()) * blockDim.x / TEAM_THREADS;
            atomicAdd(&S.mol_cyc[m], c);
            atomicAdd(&g_team_cycles[slot], (unsigned long long)c);
        }
}
__global__ void k_st_clear_cycles(State S, StagePlan Q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < Q.count && S.active[Q.mol[i]]) S.mol_cyc[Q.mol[i]] = 0.0;
}

// triangular factors of the reflector blocks in the molecule's workspace (after the filling's part)
__host__ __device__ constexpr long long stage_t_offset(int n) { return 32 + ((n + 31) & ~31); }
// workspace of a molecule's stages (doubles): the filling's part and the factors (64 x 64 per block of 64)
__host__ __device__ constexpr long long stage_workspace(int n) { return stage_t_offset(n) + (n + 63) / 64 * 4096LL; }
static_assert(stage_workspace(12) <= team_workspace(12) && stage_workspace(256) <= team_workspace(256) &&
                  stage_workspace(2405) <= team_workspace(2405),
              "a molecule's workspace has the team kernel's size");

__device__ __forceinline__ int stage_find(const long long* off, int count, long long task) {
    int lo = 0, hi = count - 1;
    while (lo < hi) {
        int mid = (lo + hi + 1) >> 1;
        if (off[mid] <= task) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------------------------- tiles
enum { ST_X = 0, ST_FP = 1, ST_C = 2, ST_P = 3, ST_W = 4 };

// One 64 x 64 tile of X, F' or W in split precision per CTA (the team GEMM on a team of as many CTAs
// as tiles: the same k-steps in the same order); W also gets its mirror image above the diagonal
// (through shared memory, both stores coalesced).
template <int MODE, bool PROF>
__global__ void __launch_bounds__(TEAM_THREADS, 2) k_st_tiles(Batch B, State S, StagePlan Q) {
    constexpr bool LOW = MODE != ST_X;
    const long long* off = LOW ? Q.off_low : Q.off_full;
    const int i = stage_find(off, Q.count, blockIdx.x), m = Q.mol[i];
    if (MODE == ST_W ? !S.conv[m] : !S.active[m]) return;
    const int n = B.m_nao[m], rt = (n + GT - 1) / GT;
    const long long mat = B.m_mat0[m];
    int tile = (int)(blockIdx.x - off[i]), bi, bj;
    if (LOW) {  // column by column from the diagonal down
        bj = 0;
        while (tile >= rt - bj) tile -= rt - bj, bj++;
        bi = bj + tile;
    } else {
        bi = rt - 1 - tile % rt;  // the rows with the longest sums first
        bj = tile / rt;
    }
    const Team t{bi + bj * rt, rt * rt, false};
    const double* Li = S.Linv + mat;
    if (MODE != ST_W) stage_start<PROF>();
    if (MODE == ST_X) {
        team_gemm(t, false, false, n, n, n, 1.0, Li, n, S.F + mat, n, 0.0, S.scr1 + mat, n, GEMM_A_LOWER | GEMM_SPLIT);
    } else if (MODE == ST_FP) {
        team_gemm(t, false, true, n, n, n, 1.0, S.scr1 + mat, n, Li, n, 0.0, S.Fp + mat, n,
                  GEMM_B_UPPER | GEMM_LOWER_TILES | GEMM_SPLIT);
    } else {
        double* out = S.W + mat;
        team_gemm(t, false, true, n, n, S.kocc[m], 1.0, S.scr1 + mat, n, S.C + mat, n, 0.0, out, n,
                  GEMM_LOWER_TILES | GEMM_SPLIT);
        for (int e = threadIdx.x; e < GT * GT; e += TEAM_THREADS) {
            int r = bi * GT + e % GT, c = bj * GT + e / GT;
            s_work[(e % GT) * (GT + 1) + e / GT] = r < n && c < n ? out[r + (long long)c * n] : 0.0;
        }
        __syncthreads();
        for (int e = threadIdx.x; e < GT * GT; e += TEAM_THREADS) {  // row of the mirror image = column here
            int c = bj * GT + e % GT, r = bi * GT + e / GT;
            if (r < n && r > c) out[c + (long long)r * n] = s_work[(e / GT) * (GT + 1) + e % GT];
        }
    }
    if (MODE != ST_W) stage_stop<PROF>(S, m, 0);
}

// The products in FP64, 32 x 32 tiles of four warps. Tiles of 64 (eight warps, two CTAs per SM) are
// bound by their SM's FP64 tensor rate where there are few (192 AOs: 18 us a stage in 9 tiles on 148
// SMs, 8 in 36 of 32; 600 AOs: 48 and 26) and have fewer warps in flight where there are many (the
// mixed batch of 1024: 7.2 ms for the four products, 6.2 in tiles of 32). The sums run over the same
// k-steps in the same order as the team GEMM's.
constexpr int G32 = 32, G32_STAGE = 2 * GK * (G32 + 2);
struct Tile32 {
    const double *A, *B;
    int lda, ldb;
    bool ta, tb;
    int M, N, k0, ke;
};
__device__ __forceinline__ void gemm_tile32(const Tile32& t, int row0, int col0, double (&acc)[2][2][2]) {
    typedef double Stage[2][GK][G32 + 2];
    Stage* stg = reinterpret_cast<Stage*>(s_work);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, wm = warp & 1, wn = warp >> 1, lr = lane >> 2, lc = lane & 3;
    const int nk = (t.ke - t.k0 + GK - 1) / GK;
    // this thread's four elements of each operand's k-step: consecutive threads along the contiguous
    // dimension, (row, k) = (am, ak) + q (ta ? (8, 0) : (0, 4)); zero outside the operands
    const int am = t.ta ? tid >> 4 : lane, ak = t.ta ? tid & 15 : warp, bn = t.tb ? lane : tid >> 4, bk = t.tb ? warp : tid & 15;
    const double* pa = t.A + (t.ta ? t.k0 + ak + (long long)(row0 + am) * t.lda : row0 + am + (long long)(t.k0 + ak) * t.lda);
    const double* pb = t.B + (t.tb ? col0 + bn + (long long)(t.k0 + bk) * t.ldb : t.k0 + bk + (long long)(col0 + bn) * t.ldb);
    const long long qa = (t.ta ? 8LL : 4LL) * t.lda, qb = (t.tb ? 4LL : 8LL) * t.ldb;
    const long long sa = t.ta ? GK : (long long)GK * t.lda, sb = t.tb ? (long long)GK * t.ldb : GK;
    auto issue = [&](int ks) {
        if (ks < nk) {
            Stage& S = stg[ks % GSTAGES];
            const int left = t.ke - t.k0 - ks * GK;  // k's left from this step on
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int mm = t.ta ? am + 8 * q : am, kk = t.ta ? ak : ak + 4 * q;
                const bool ok = row0 + mm < t.M && kk < left;
                cp_async8(&S[0][kk][mm], ok ? pa + q * qa : t.A, ok);
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int nn = t.tb ? bn : bn + 8 * q, kk = t.tb ? bk + 4 * q : bk;
                const bool ok = col0 + nn < t.N && kk < left;
                cp_async8(&S[1][kk][nn], ok ? pb + q * qb : t.B, ok);
            }
            pa += sa;
            pb += sb;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) acc[i][j][0] = acc[i][j][1] = 0.0;
    for (int ks = 0; ks < GSTAGES - 1; ks++) issue(ks);
    for (int ks = 0; ks < nk; ks++) {
        cp_async_wait<GSTAGES - 2>();
        __syncthreads();
        issue(ks + GSTAGES - 1);
        Stage& S = stg[ks % GSTAGES];
#pragma unroll
        for (int kk = 0; kk < GK; kk += 4) {
            double af[2], bf[2];
#pragma unroll
            for (int i = 0; i < 2; i++) af[i] = S[0][kk + lc][wm * 16 + i * 8 + lr];
#pragma unroll
            for (int j = 0; j < 2; j++) bf[j] = S[1][kk + lc][wn * 16 + j * 8 + lr];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
}

template <int MODE, bool PROF>
__global__ void __launch_bounds__(128) k_st_tiles32(Batch B, State S, StagePlan Q) {
    constexpr bool LOW = MODE == ST_FP || MODE == ST_P || MODE == ST_W;
    const long long* off = LOW ? Q.off_low32 : Q.off_full32;
    const int i = stage_find(off, Q.count, blockIdx.x), m = Q.mol[i];
    if (MODE == ST_W ? !S.conv[m] : !S.active[m]) return;
    const int n = B.m_nao[m], rt = (n + G32 - 1) / G32, ao0 = B.m_ao0[m];
    const long long mat = B.m_mat0[m];
    int tile = (int)(blockIdx.x - off[i]), bi, bj;
    if (LOW) {
        bj = 0;
        while (tile >= rt - bj) tile -= rt - bj, bj++;
        bi = bj + tile;
    } else {
        bi = rt - 1 - tile % rt;
        bj = tile / rt;
    }
    const int k = MODE >= ST_C ? S.kocc[m] : n, row0 = bi * G32, col0 = bj * G32;
    if (MODE == ST_C && col0 >= k) return;
    if (MODE != ST_W) stage_start<PROF>();
    const double* Li = S.Linv + mat;
    double* out;
    Tile32 t;
    if (MODE == ST_X) {
        t = {Li, S.F + mat, n, n, false, false, n, n, 0, min(n, row0 + G32)};
        out = S.scr1 + mat;
    } else if (MODE == ST_FP) {
        t = {S.scr1 + mat, Li, n, n, false, true, n, n, 0, min(n, col0 + G32)};
        out = S.Fp + mat;
    } else if (MODE == ST_C) {
        t = {Li, S.Z + mat, n, n, true, false, n, k, row0, n};
        out = S.C + mat;
    } else {
        t = {S.scr1 + mat, S.C + mat, n, n, false, true, n, n, 0, k};
        out = (MODE == ST_P ? S.P : S.W) + mat;
    }
    double acc[2][2][2];
    gemm_tile32(t, row0, col0, acc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3;
#pragma unroll
    for (int x = 0; x < 2; x++)
#pragma unroll
        for (int y = 0; y < 2; y++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = row0 + (warp & 1) * 16 + x * 8 + lr, c = col0 + (warp >> 1) * 16 + y * 8 + lc * 2 + h;
                if (r >= n || c >= t.N) continue;
                const double v = acc[x][y][h];
                if (MODE == ST_P || MODE == ST_W) {  // the lower triangle and its mirror image
                    if (r < c) continue;
                    out[c + (long long)r * n] = v;
                }
                out[r + (long long)c * n] = v;
                if (MODE == ST_C) S.scr1[mat + r + (long long)c * n] = v * S.focc[ao0 + c];
            }
    if (MODE != ST_W) stage_stop<PROF>(S, m, MODE == ST_C ? 6 : MODE == ST_P ? 7 : 0);
}

// scr1 = C (f e), the left factor of W
__global__ void k_st_scale(Batch B, State S, StagePlan Q) {
    const int i = stage_find(Q.off_full, Q.count, blockIdx.x), m = Q.mol[i];
    if (!S.conv[m]) return;
    const int n = B.m_nao[m], rt = (n + GT - 1) / GT, ao0 = B.m_ao0[m], k = S.kocc[m];
    const int tile = (int)(blockIdx.x - Q.off_full[i]), bi = tile % rt, bj = tile / rt;
    const long long mat = B.m_mat0[m];
    for (int e = threadIdx.x; e < GT * GT; e += blockDim.x) {
        int r = bi * GT + e % GT, c = bj * GT + e / GT;
        long long a = mat + r + (long long)c * n;
        if (r < n && c < k) S.scr1[a] = S.C[a] * (S.focc[ao0 + c] * S.emo[ao0 + c]);
    }
}

// ---------------------------------------------------------------------------------- orbital energies
// Number of eigenvalues below x of the tridiagonal matrix de[i] = (d_i, e_{i-1}^2), padded to a
// multiple of sixteen rows beyond the first. The Sturm sequence as determinants of the leading
// blocks, p_i = (d_i - x) p_{i-1} - e^2 p_{i-2}, counting sign changes: one FMA per row on the
// dependent chain (11 cycles) where the quotients q_i = p_i / p_{i-1} take a division (~120). Every
// sixteen rows the pair is scaled by a power of two; a block in which it vanished (a zero pivot
// followed by a zero coupling) is done again with the quotients and their pivot floor.
constexpr int ST_ROWS = 16;
__device__ __forceinline__ int sturm_det(const double2* de, int nb, double x, double pivmin) {
    double p0 = 1.0, p1 = de[0].x - x;
    int cnt = p1 < 0.0;
    for (int b = 0; b < nb; b++) {
        const double2* w = de + 1 + ST_ROWS * b;
        const double s0 = p0, s1 = p1;
        const int c0 = cnt;
#pragma unroll
        for (int u = 0; u < ST_ROWS; u++) {
            double p2 = fma(w[u].x - x, p1, -(w[u].y * p0));
            cnt += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
            p0 = p1;
            p1 = p2;
        }
        const double a = fmax(fabs(p0), fabs(p1));
        if (a > 1e-200 && a < 1e200) {
            const double s = __hiloint2double((2046 - (__double2hiint(a) >> 20)) << 20, 0);
            p0 *= s;
            p1 *= s;
        } else {
            double q = s0 != 0.0 ? s1 / s0 : copysign(INFINITY, s1);
            cnt = c0;
            for (int u = 0; u < ST_ROWS; u++) {
                q = w[u].x - x - w[u].y / q;
                if (fabs(q) < pivmin) q = -pivmin;
                cnt += q < 0.0;
            }
            const bool big = fabs(q) > 1e100;
            p0 = big ? 1.0 / fabs(q) : 1.0;
            p1 = big ? copysign(1.0, q) : q;
        }
    }
    return cnt;
}

// d, e^2 of a tridiagonal matrix in shared memory (sturm_det's form), its Gershgorin bounds and
// pivot floor (the same values as team_gershgorin's); returns the number of 16-row blocks
__device__ int cta_tridiagonal(const double* d, const double* e, int n, double2* de, double* g) {
    __shared__ double slo[TEAM_THREADS / 32], shi[TEAM_THREADS / 32], sem[TEAM_THREADS / 32];
    double lo = INFINITY, hi = -INFINITY, emax = 0.0;
    const int nb = (n - 1 + ST_ROWS - 1) / ST_ROWS;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        double el = i > 0 ? e[i - 1] : 0.0, er = i + 1 < n ? e[i] : 0.0, di = d[i];
        double r = fabs(el) + fabs(er);
        lo = fmin(lo, di - r);
        hi = fmax(hi, di + r);
        emax = fmax(emax, el * el);
        de[i] = make_double2(di, el * el);
    }
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        emax = fmax(emax, __shfl_xor_sync(0xffffffffu, emax, o));
    }
    const int w = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) slo[w] = lo, shi[w] = hi, sem[w] = emax;
    __syncthreads();
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) {
        lo = fmin(lo, slo[q]);
        hi = fmax(hi, shi[q]);
        emax = fmax(emax, sem[q]);
    }
    double tnrm = fmax(fabs(lo), fabs(hi));
    g[0] = lo - (2.0 * DBL_EPSILON * tnrm * n + 1e-300);
    g[1] = hi + (2.0 * DBL_EPSILON * tnrm * n + 1e-300);
    g[2] = DBL_MIN * fmax(1.0, emax);
    // padding rows: above every shift, uncoupled, so no sign changes
    for (int i = n + threadIdx.x; i < 1 + ST_ROWS * nb; i += blockDim.x) de[i] = make_double2(g[1] + 1.0, 0.0);
    __syncthreads();
    return nb;
}

// The levels k0 + (thread / 4) below k1 of one tridiagonal matrix, four threads a level: the counts
// at 128 points of the Gershgorin interval bracket every level, then each group cuts its bracket
// into five per pass (21 passes over the matrix where bisection takes 55: at one molecule the
// passes are a latency chain, and a full batch has the issue slots to spare).
constexpr int ST_POINTS = 128;
__device__ void cta_levels(const double2* de, int nb, const double* g, int k0, int k1, double* w) {
    __shared__ int cnt[ST_POINTS];
    const int tid = threadIdx.x;
    const double step = (g[1] - g[0]) * (1.0 / (ST_POINTS + 1));
    if (tid < ST_POINTS) cnt[tid] = sturm_det(de, nb, g[0] + step * (tid + 1), g[2]);
    __syncthreads();
    const int k = k0 + (tid >> 2), sub = tid & 3;
    bool live = k < k1;
    int a = 0, b = ST_POINTS;  // smallest point with a count above k
    while (a < b) {
        int mid = (a + b) >> 1;
        if (cnt[mid] > k) b = mid;
        else a = mid + 1;
    }
    double lo = a > 0 ? g[0] + step * a : g[0], hi = a < ST_POINTS ? g[0] + step * (a + 1) : g[1];
    for (int it = 0; it < 200; it++) {
        double wd = hi - lo;
        if (bisect_done(lo, hi, g[2]) || lo + 0.2 * wd <= lo || lo + 0.8 * wd >= hi) live = false;
        if (!__any_sync(0xffffffffu, live)) break;
        int below = 0;
        if (live) below = sturm_det(de, nb, lo + (0.2 * (sub + 1)) * wd, g[2]) <= k;
        // points of the group that lie below the level
        unsigned bits = __ballot_sync(0xffffffffu, below) >> (tid & 28) & 15u;
        int t = __popc(bits);
        if (live) {
            double l = lo;
            if (t > 0) lo = l + (0.2 * t) * wd;
            if (t < 4) hi = l + (0.2 * (t + 1)) * wd;
        }
    }
    if (k < k1 && sub == 0) w[k] = 0.5 * (lo + hi);
    __syncthreads();
}

__device__ __forceinline__ int first_levels(const Batch& B, int m, int n) {
    return min(n, (int)ceil(fmax(B.m_nalpha[m], B.m_nbeta[m])) + max(16, n / 16));
}

// 32 levels per CTA (128 threads: one warp per scheduler, so that the chain's latency and not its
// issue slots set the time of a single molecule). The SCF takes the lowest ceil(n_occ) + max(16,
// n/16) and gives the others the Gershgorin bound; rest: those others (every orbital energy of the
// result).
template <bool PROF>
__global__ void __launch_bounds__(ST_POINTS) k_st_bisect(Batch B, State S, StagePlan Q, int rest) {
    const int i = stage_find(Q.off_vec, Q.count, blockIdx.x), m = Q.mol[i];
    if (!rest && !S.active[m]) return;
    const int n = B.m_nao[m], ao0 = B.m_ao0[m], kc = first_levels(B, m, n);
    const int k0 = 32 * (int)(blockIdx.x - Q.off_vec[i]), k1 = min(n, k0 + 32);
    const int lo = rest ? max(k0, kc) : k0, hi = rest ? k1 : min(k1, kc);
    if (rest && lo >= hi) return;
    if (!rest) stage_start<PROF>();
    double2* de = reinterpret_cast<double2*>(s_work);
    double g[3];
    int nb = cta_tridiagonal(S.dtri + ao0, S.etri + ao0, n, de, g);
    if (lo < hi) cta_levels(de, nb, g, lo, hi, S.emo + ao0);
    if (!rest)
        for (int k = max(k0, kc) + threadIdx.x; k < k1; k += blockDim.x) S.emo[ao0 + k] = g[1];
    if (!rest) stage_stop<PROF>(S, m, 2);
}

// ---------------------------------------------------------------------------------- filling
// tblite's Fermi filling (mol_fermi: the same sums in the same order; with equal spins the second
// filling is the first, and a level with 0 or 1 electrons has no entropy). When the last computed
// level still holds electrons, the CTA computes the others and fills again.
template <bool PROF>
__global__ void __launch_bounds__(TEAM_THREADS) k_st_fermi(Batch B, State S, StagePlan Q) {
    const int m = Q.mol[blockIdx.x];
    if (!S.active[m]) return;
    stage_start<PROF>();
    const int n = B.m_nao[m], ao0 = B.m_ao0[m], lane = threadIdx.x & 31;
    const double na = B.m_nalpha[m], nbeta = B.m_nbeta[m];
    double* focc = S.focc + ao0;
    __shared__ int s_more;
    double2* de = reinterpret_cast<double2*>(s_work);
    double* emo = s_work;  // staged levels, alpha and beta occupations
    double *oa = s_work + n, *ob = s_work + 2 * n;
    int kc = first_levels(B, m, n);
    for (int round = 0; round < 2; round++) {
        for (int k = threadIdx.x; k < n; k += blockDim.x) emo[k] = S.emo[ao0 + k];
        __syncthreads();
        if (threadIdx.x < 32) {
            double efa, efb;
            warp_fill(na, B.kt, emo, n, oa, &efa);
            if (nbeta == na) {
                efb = efa;
                for (int k = lane; k < n; k += 32) ob[k] = oa[k];
            } else warp_fill(nbeta, B.kt, emo, n, ob, &efb);
            __syncwarp();
            double pa = 0.0, pb = 0.0, ts = 0.0, flast = 0.0;
            int kl = 0;
            auto entropy = [](double f) { return f == 0.0 || f == 1.0 ? 0.0 : log(pow(f, f) * pow(1.0 - f, 1.0 - f)); };
            for (int k = lane; k < n; k += 32) {
                double fa = oa[k], fb = ob[k];
                if (S.focc_a) S.focc_a[ao0 + k] = fa;
                pa += fa;
                pb += fb;
                if (B.kt > 0.0) {
                    double sa = entropy(fa);
                    ts += sa + (fb == fa ? sa : entropy(fb));
                }
                if (k == kc - 1) flast = fmax(fa, fb);
                double f = fa + fb;
                focc[k] = f;
                if (f > 1e-16) kl = max(kl, k + 1);
            }
            pa = warp_sum(pa);
            pb = warp_sum(pb);
            ts = warp_sum(ts);
            for (int o = 16; o > 0; o >>= 1) {
                kl = max(kl, __shfl_xor_sync(0xffffffffu, kl, o));
                flast = fmax(flast, __shfl_xor_sync(0xffffffffu, flast, o));
            }
            if (lane == 0) {
                S.kocc[m] = kl;
                S.ts[m] = ts * B.kt;
                if (S.efermi) {  // the Fermi levels, NaN where the filling is aufbau (0 K, no electrons)
                    const double nan = __longlong_as_double(0x7ff8000000000000LL);
                    S.efermi[2 * m] = B.kt > 0.0 && na > 0.0 ? efa : nan;
                    S.efermi[2 * m + 1] = B.kt > 0.0 && nbeta > 0.0 ? efb : nan;
                }
                s_more = kc < n && flast > 1e-16;
                if (fabs(pa - na) > 1e-6 || fabs(pb - nbeta) > 1e-6) atomicOr(&S.status[m], ST_FERMI);
            }
        }
        __syncthreads();
        if (!s_more) break;
        double g[3];
        int nb = cta_tridiagonal(S.dtri + ao0, S.etri + ao0, n, de, g);
        for (int k0 = kc; k0 < n; k0 += 64) cta_levels(de, nb, g, k0, min(n, k0 + 64), S.emo + ao0);
        kc = n;
    }
    stage_stop<PROF>(S, m, 3);
}

// ---------------------------------------------------------------------------------- vectors
// Inverse iteration as in team_invit (two solves from a hashed start; the vectors of a cluster, closer
// than 1e-6 ||T||, made orthogonal after each), one thread per vector, 32 per CTA: part 0 factorises
// and solves (twice for a vector outside the clusters), part 1 solves again for the clusters' vectors,
// each followed by k_st_gs (one thread took a whole cluster before, and a launch was as long as its
// largest). The first forward substitution
// rides on the factorisation, the factors hold reciprocal pivots (one division per row instead of
// three), norms are summed as the solution is made and applied by the next reader, and rows come
// through a ring of asynchronous copies, 28 ahead. The vectors stay where they are made,
// row-interleaved in the P plane ([row * n + vector]).
struct Clusters {  // the clusters of a molecule's levels and the shifts of the solves
    double ctol, pert, pivmin;
};
// by one warp: ||T|| and what follows from it
__device__ __forceinline__ Clusters warp_clusters(const double* d, const double* e, int n) {
    double tnrm = 0.0;
    for (int i = threadIdx.x & 31; i < n; i += 32)
        tnrm = fmax(tnrm, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + (i + 1 < n ? fabs(e[i]) : 0.0));
    for (int o = 16; o > 0; o >>= 1) tnrm = fmax(tnrm, __shfl_xor_sync(0xffffffffu, tnrm, o));
    if (tnrm == 0.0) tnrm = 1.0;
    return {1e-6 * tnrm, 10.0 * DBL_EPSILON * tnrm, DBL_EPSILON * tnrm};
}

// a pivot whose reciprocal is finite: a zero or subnormal one becomes the floor
__device__ __forceinline__ double invit_pivot(double pv, double floor) { return fabs(pv) < DBL_MIN ? floor : pv; }

__host__ __device__ constexpr int st_invit_bytes(int n) { return 8 * (2 * (n + 8) + 32 * 3 * 32); }
__device__ __forceinline__ double* stage_norms(const TeamPlan& P, int m) { return P.wk + P.m_wk0[m] + 32; }

template <bool PROF>
__global__ void __launch_bounds__(32) k_st_invit(Batch B, State S, StagePlan Q, TeamPlan P, int part) {
    const int ti = stage_find(Q.off_vec, Q.count, blockIdx.x), m = Q.mol[ti];
    if (!S.active[m]) return;
    const int n = B.m_nao[m], ao0 = B.m_ao0[m], k = S.kocc[m];
    const int q = 32 * (int)(blockIdx.x - Q.off_vec[ti]) + threadIdx.x;
    if (q - (int)threadIdx.x >= k) return;
    stage_start<PROF>();
    const long long mat = B.m_mat0[m], LD = n;
    const double* w = S.emo + ao0;
    double *sd = s_work, *se = s_work + n + 8;  // the tridiagonal matrix (e: two rows of zeros beyond)
    for (int i = threadIdx.x; i < n + 8; i += 32) {
        sd[i] = i < n ? S.dtri[ao0 + i] : 0.0;
        se[i] = i + 1 < n ? S.etri[ao0 + i] : 0.0;
    }
    __syncwarp();
    const Clusters cl = warp_clusters(sd, se, n);
    // alone: no level close by, so nothing to be made orthogonal to, and part 0 takes both solves
    const bool alone = q < k && !(q > 0 && w[q] - w[q - 1] <= cl.ctol) && !(q + 1 < k && w[q + 1] - w[q] <= cl.ctol);
    const bool works = q < k && !(part == 1 && alone);
    int first = 0;  // keeps the time
    if constexpr (PROF) first = __ffs(__ballot_sync(0xffffffffu, works)) - 1;
    if (!works) return;
    double* u0 = S.scr1 + mat + q;  // reciprocal pivots
    double* u1 = S.scr2 + mat + q;
    double* lm = S.scr3 + mat + q;
    double* x = S.P + mat + q;
    unsigned* swaps = reinterpret_cast<unsigned*>(S.piv + mat) + q;  // a bit per row, a word per 32 rows
    // the thread's own ring of rows on their way from L2 or HBM
    constexpr int GR = 4, NG = 8, R = GR * NG;
    double* ring = s_work + 2 * (n + 8) + threadIdx.x;
    auto slot = [&](int step, int f) { return ring + ((step & (R - 1)) * 3 + f) * 32; };  // f beyond 2: later rows
    double nrm = 1.0;  // 1 / norm of the last solution
    // L with the row interchanges, the first solution (1 / its norm: nr) normalised on the way
    auto forward = [&](double nr) {
        const long long st = LD;
        auto issue = [&](int g) {
            const double *px = x + (g * GR + 1) * st, *pl = lm + g * GR * st;
            if (g * GR + GR < n) {
#pragma unroll
                for (int u = 0; u < GR; u++, px += st, pl += st) {
                    cp_async8(slot(g * GR, 3 * u), px, true);
                    cp_async8(slot(g * GR, 3 * u + 1), pl, true);
                }
            } else {
                for (int u = 0; g * GR + u + 1 < n; u++, px += st, pl += st) {
                    cp_async8(slot(g * GR, 3 * u), px, true);
                    cp_async8(slot(g * GR, 3 * u + 1), pl, true);
                }
            }
            cp_async_commit();
        };
        double cur = x[0] * nr;
        unsigned bits = 0;
        for (int g = 0; g < NG - 1; g++) issue(g);
        double* px = x;
        for (int g = 0; g * GR + 1 < n; g++) {
            cp_async_wait<NG - 2>();
            if ((g * GR & 31) == 0) bits = swaps[(g * GR >> 5) * st];
            double xv[GR], l[GR];
#pragma unroll
            for (int u = 0; u < GR; u++) xv[u] = *slot(g * GR, 3 * u), l[u] = *slot(g * GR, 3 * u + 1);
            issue(g + NG - 1);
#pragma unroll
            for (int u = 0; u < GR; u++) {
                if (g * GR + u + 1 < n) {
                    const bool p = bits & 1;
                    bits >>= 1;
                    const double nxt = xv[u] * nr, top = p ? nxt : cur;
                    *px = top;
                    px += st;
                    cur = (p ? cur : nxt) - l[u] * top;
                }
            }
        }
        cp_async_wait<0>();
        x[(n - 1) * st] = cur;
    };
    // U with up to two superdiagonals (e_{i+1} after an interchange); its norm's reciprocal into nrm
    auto backward = [&]() {
        const long long st = LD;
        auto issue = [&](int g) {  // rows n - 1 - 4 g downwards
            const long long o = (n - 1 - g * GR) * st;
            const double *px = x + o, *p0 = u0 + o, *p1 = u1 + o;
            const int cnt = min(GR, n - g * GR);
            if (cnt == GR) {
#pragma unroll
                for (int u = 0; u < GR; u++, px -= st, p0 -= st, p1 -= st) {
                    cp_async8(slot(g * GR, 3 * u), px, true);
                    cp_async8(slot(g * GR, 3 * u + 1), p0, true);
                    cp_async8(slot(g * GR, 3 * u + 2), p1, true);
                }
            } else {
                for (int u = 0; u < cnt; u++, px -= st, p0 -= st, p1 -= st) {
                    cp_async8(slot(g * GR, 3 * u), px, true);
                    cp_async8(slot(g * GR, 3 * u + 1), p0, true);
                    cp_async8(slot(g * GR, 3 * u + 2), p1, true);
                }
            }
            cp_async_commit();
        };
        double xn1 = 0.0, xn2 = 0.0, ss = 0.0;
        for (int g = 0; g < NG - 1; g++) issue(g);
        unsigned bits = swaps[((n - 1) >> 5) * st] << (31 - ((n - 1) & 31));
        double* px = x + (n - 1) * st;
        for (int g = 0; g * GR < n; g++) {
            cp_async_wait<NG - 2>();
            double xv[GR], f0[GR], f1[GR];
#pragma unroll
            for (int u = 0; u < GR; u++) {
                xv[u] = *slot(g * GR, 3 * u);
                f0[u] = *slot(g * GR, 3 * u + 1);
                f1[u] = *slot(g * GR, 3 * u + 2);
            }
            issue(g + NG - 1);
#pragma unroll
            for (int u = 0; u < GR; u++) {
                const int i = n - 1 - (g * GR + u);
                if (i >= 0) {
                    if ((i & 31) == 31) bits = swaps[(i >> 5) * st];
                    const double c1 = i + 1 < n ? f1[u] : 0.0, c2 = i + 2 < n && (int)bits < 0 ? se[i + 1] : 0.0;
                    bits <<= 1;
                    double v = fma(-c1, xn1, fma(-c2, xn2, xv[u])) * f0[u];
                    *px = v;
                    px -= st;
                    xn2 = xn1;
                    xn1 = v;
                    ss = fma(v, v, ss);
                }
            }
        }
        cp_async_wait<0>();
        nrm = 1.0 / sqrt(ss);
        if (!(ss > 1e-280 && ss < INFINITY)) {
            // the squares left the range (a level within 1e-140 of a decoupled row's diagonal element gives
            // elements above 1e154), not the solution: its norm from elements scaled by the largest
            double mx = 0.0, sc = 0.0;
            for (int i = 0; i < n; i++) mx = fmax(mx, fabs(x[i * st]));
            const double inv = 1.0 / mx;
            for (int i = 0; i < n; i++) sc = fma(x[i * st] * inv, x[i * st] * inv, sc);
            nrm = inv / sqrt(sc);
            if (isnan(ss) || !(mx > 0.0 && mx < INFINITY)) {
                atomicOr(&S.status[m], ST_INVIT);
                nrm = 1.0;
            }
        }
    };
    if (part == 0) {
        // the shift: the level, kept apart from the cluster's earlier ones
        int q0 = q;
        while (q0 > 0 && w[q0] - w[q0 - 1] <= cl.ctol) q0--;
        double lam = w[q0];
        for (int p = q0 + 1; p <= q; p++) lam = fmax(w[p], lam + cl.pert);
        // LU with partial pivoting of T - lam I, the start vector eliminated along
        double ca = sd[0] - lam, cb = se[0];
        unsigned bits = 0;
        double cur = hash_uniform((unsigned)q, 0u);
#pragma unroll 4
        for (int i = 0; i + 1 < n; i++) {
            const double sub = se[i], a1 = sd[i + 1] - lam, b1 = se[i + 1];
            const double nxt = hash_uniform((unsigned)q, (unsigned)(i + 1));
            const bool p = fabs(ca) < fabs(sub);
            const double pv = invit_pivot(p ? sub : ca, cl.pivmin);
            const double inv = 1.0 / pv, l = (p ? ca : sub) * inv, t1 = p ? a1 : cb;
            const long long ix = (long long)i * LD;
            u0[ix] = inv;
            u1[ix] = t1;
            lm[ix] = l;
            x[ix] = p ? nxt : cur;
            bits |= (unsigned)p << (i & 31);
            if ((i & 31) == 31) {
                swaps[(i >> 5) * LD] = bits;
                bits = 0;
            }
            cur = (p ? cur : nxt) - l * (p ? nxt : cur);
            ca = (p ? cb : a1) - l * t1;
            cb = p ? -l * b1 : b1;
        }
        swaps[((n - 1) >> 5) * LD] = bits;
        u0[(n - 1) * LD] = 1.0 / invit_pivot(ca, cl.pivmin);
        x[(n - 1) * LD] = cur;
        backward();
        if (alone) {
            forward(nrm);
            backward();
        }
    } else {
        forward(stage_norms(P, m)[q]);
        backward();
    }
    stage_norms(P, m)[q] = nrm;  // applied by whoever reads the vector next
    stage_stop<PROF>(S, m, 4, first);
}

// Gram-Schmidt within the clusters (ascending, each vector against all earlier ones of its cluster,
// then normalised), a warp per cluster: the warp of block q's 32 levels takes the clusters whose
// first level lies there.
template <bool PROF>
__global__ void __launch_bounds__(32) k_st_gs(Batch B, State S, StagePlan Q, TeamPlan P) {
    const int ti = stage_find(Q.off_vec, Q.count, blockIdx.x), m = Q.mol[ti];
    if (!S.active[m]) return;
    const int n = B.m_nao[m], ao0 = B.m_ao0[m], k = S.kocc[m], lane = threadIdx.x;
    const int qb = 32 * (int)(blockIdx.x - Q.off_vec[ti]);
    if (qb >= k) return;
    stage_start<PROF>();
    const double* w = S.emo + ao0;
    const Clusters cl = warp_clusters(S.dtri + ao0, S.etri + ao0, n);
    // heads: not close to the level below, close to the level above
    const int q = qb + lane;
    const bool head = q + 1 < k && w[q + 1] - w[q] <= cl.ctol && !(q > 0 && w[q] - w[q - 1] <= cl.ctol);
    unsigned heads = __ballot_sync(0xffffffffu, head);
    double* x = S.P + B.m_mat0[m];
    while (heads) {
        const int q0 = qb + __ffs(heads) - 1;
        heads &= heads - 1;
        double* norm = stage_norms(P, m);
        const double nh = norm[q0];
        for (int i = lane; i < n; i += 32) x[(long long)i * n + q0] *= nh;
        __syncwarp();
        if (lane == 0) norm[q0] = 1.0;
        for (int q1 = q0 + 1; q1 < k && w[q1] - w[q1 - 1] <= cl.ctol; q1++) {
            double ss = 0.0, nq = norm[q1];  // the norm goes in with the first projection
            __syncwarp();
            if (lane == 0) norm[q1] = 1.0;
            for (int p = q0; p < q1; p++) {
                double dt = 0.0;
#pragma unroll 4
                for (int i = lane; i < n; i += 32) dt = fma(x[(long long)i * n + p], x[(long long)i * n + q1] * nq, dt);
                dt = warp_sum(dt);
                ss = 0.0;
                for (int i0 = lane; i0 < n; i0 += 128) {
                    double a[4], c[4];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const long long r = (long long)min(i0 + 32 * u, n - 1) * n;
                        a[u] = x[r + p];
                        c[u] = x[r + q1];
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (i0 + 32 * u < n) {
                            double v = fma(-dt, a[u], c[u] * nq);
                            x[(long long)(i0 + 32 * u) * n + q1] = v;
                            ss = fma(v, v, ss);
                        }
                }
                nq = 1.0;
            }
            ss = warp_sum(ss);
            const double nr = 1.0 / sqrt(ss);
            for (int i0 = lane; i0 < n; i0 += 128) {
                double c[4];
#pragma unroll
                for (int u = 0; u < 4; u++) c[u] = x[(long long)min(i0 + 32 * u, n - 1) * n + q1];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i0 + 32 * u < n) x[(long long)(i0 + 32 * u) * n + q1] = c[u] * nr;
            }
        }
    }
    stage_stop<PROF>(S, m, 4);
}

// ---------------------------------------------------------------------------------- back-transformation
constexpr int ST_NB = 64;  // reflectors per block

// T of block b: H_{64 b} H_{64 b + 1} .. = I - V T V^T (T upper triangular; column c is
// -tau_c T[0:c, 0:c] (V^T V)[0:c, c]), four threads per row
template <bool PROF>
__global__ void __launch_bounds__(TEAM_THREADS) k_st_tfac(Batch B, State S, StagePlan Q, TeamPlan P) {
    const int i = stage_find(Q.off_rt, Q.count, blockIdx.x), m = Q.mol[i];
    if (!S.active[m]) return;
    const int n = B.m_nao[m], b0 = ST_NB * (int)(blockIdx.x - Q.off_rt[i]), jb = min(ST_NB, n - 2 - b0);
    if (jb <= 0) return;
    stage_start<PROF>();
    const double* V = S.Fp + B.m_mat0[m];
    double* T = P.wk + P.m_wk0[m] + stage_t_offset(n) + (long long)(b0 / ST_NB) * ST_NB * ST_NB;
    const Team t{0, 1, false};
    const double* Vb = V + b0 + (long long)b0 * n;  // rows from b0 on: nothing above
    team_gemm(t, true, false, jb, jb, n - b0, 1.0, Vb, n, Vb, n, 0.0, T, ST_NB);
    __syncthreads();
    constexpr int LT = ST_NB + 1;
    double *sg = s_work, *st = s_work + ST_NB * LT;
    for (int e = threadIdx.x; e < ST_NB * ST_NB; e += blockDim.x) {
        int r = e % ST_NB, c = e / ST_NB;
        sg[c * LT + r] = r < jb && c < jb ? T[r + c * ST_NB] : 0.0;
        st[c * LT + r] = 0.0;
    }
    __syncthreads();
    const int r = threadIdx.x >> 2, sub = threadIdx.x & 3;
    for (int c = 0; c < jb; c++) {
        const double tc = S.tau[B.m_ao0[m] + b0 + c];
        double s = 0.0;
        for (int q = r + sub; q < c; q += 4) s += st[q * LT + r] * sg[c * LT + q];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        if (sub == 0) st[c * LT + r] = r < c ? -tc * s : r == c ? tc : 0.0;
        __syncthreads();
    }
    for (int e = threadIdx.x; e < ST_NB * ST_NB; e += blockDim.x) T[e] = st[(e / ST_NB) * LT + e % ST_NB];
    stage_stop<PROF>(S, m, 5);
}

// shared memory of k_st_apply (doubles): the columns, row by row, then three 64 x NC blocks. NC is 8
// or 24: a row pitch of 8 mod 16 doubles serves the fragments without bank conflicts as it is.
__host__ __device__ constexpr long long st_apply_doubles(int n, int nc) { return (long long)((n + 7) / 8 * 8 + 3 * ST_NB) * nc; }
// the most AOs whose columns fit so many bytes
__host__ __device__ constexpr int st_apply_rows(int nc, int bytes) { return (bytes / 8 / nc - 3 * ST_NB) / 8 * 8; }
constexpr int ST_SMEM_MAX = TRD_SMEM_MAX - 512;  // dynamic, of the stages' kernels (they have some of their own)
static_assert(st_apply_doubles(st_apply_rows(24, ST_SMEM_MAX), 24) * 8 <= ST_SMEM_MAX &&
              st_apply_doubles(st_apply_rows(24, ST_SMEM_MAX) + 1, 24) * 8 > ST_SMEM_MAX,
              "st_apply_rows is st_apply_doubles' inverse");

// Z <- Q Z for NC columns, held in shared memory from the first block of reflectors to the last:
// per block Y = V^T Z, Y <- T Y, Z -= V Y on the FP64 tensor cores, V straight from L2 into the
// fragments. Y's sum over the rows runs in halves (row / 64 mod 2) of four interleaved chains (row / 4
// mod 4), added in order: by 16 warps at once, or by 8 one half after the other (two CTAs per SM).
template <int NC, int NW, bool PROF>
__global__ void __launch_bounds__(32 * NW, NW == 8 ? 2 : 1) k_st_apply(Batch B, State S, StagePlan Q, TeamPlan P, int n_lo, int n_hi) {
    constexpr int NT = NC / 8, LP = NC;
    static_assert(NC % 16 == 8, "row pitch");
    const int ti = stage_find(Q.off_col, Q.count, blockIdx.x), m = Q.mol[ti];
    if (!S.active[m] || Q.width[ti] != NC) return;
    const int n = B.m_nao[m], k = S.kocc[m], c0 = NC * (int)(blockIdx.x - Q.off_col[ti]);
    if (c0 >= k || n <= n_lo || n > n_hi) return;  // another launch's molecules: each asks for its own shared memory
    stage_start<PROF>();
    const long long mat = B.m_mat0[m];
    const int n8 = (n + 7) / 8 * 8, nrefl = n - 2;
    double* z = s_work;
    double* ya = z + (long long)n8 * LP;
    double* yh = ya + ST_NB * LP;
    double* yb = yh + ST_NB * LP;
    const double* V = S.Fp + mat;
    const double* X = S.P + mat;
    const double* T0 = P.wk + P.m_wk0[m] + stage_t_offset(n);
    const double* norm = stage_norms(P, m);
    for (int e = threadIdx.x; e < n8 * NC; e += blockDim.x) {
        int r = e / NC, c = e % NC;
        z[r * LP + c] = r < n && c0 + c < k ? X[(long long)r * n + c0 + c] * norm[c0 + c] : 0.0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lr = lane >> 2, lc = lane & 3, mt = warp & 7;
    for (int b0 = (nrefl - 1) / ST_NB * ST_NB; b0 >= 0; b0 -= ST_NB) {
        const int jb = min(ST_NB, nrefl - b0);
        // Y: eight reflectors per warp (one per lane group of four), rows from b0 on (zeros above b0 + 1)
        for (int hf = warp >> 3; hf < 2; hf += NW / 8) {
            const int c = b0 + 8 * mt + lr;
            const bool in = 8 * mt + lr < jb;
            const double* vc = V + (long long)(in ? c : b0) * n;
            double acc[4][NT][2];
#pragma unroll
            for (int s = 0; s < 4; s++)
#pragma unroll
                for (int t = 0; t < NT; t++) acc[s][t][0] = acc[s][t][1] = 0.0;
            for (int r0 = b0 + 64 * hf; r0 < n; r0 += 128) {  // sixteen loads in flight per lane
                double a[16];
#pragma unroll
                for (int s = 0; s < 16; s++) {
                    int r = r0 + 4 * s + lc;
                    a[s] = in && r < n ? vc[r] : 0.0;
                }
#pragma unroll
                for (int s = 0; s < 16; s++) {
                    const int rb = r0 + 4 * s;
                    if (rb >= n8) break;
                    const double* zr = z + (rb + lc) * LP + lr;
#pragma unroll
                    for (int t = 0; t < NT; t++) dmma_8x8x4(acc[s & 3][t][0], acc[s & 3][t][1], a[s], zr[8 * t]);
                }
            }
            double* dst = hf ? yh : ya;
#pragma unroll
            for (int t = 0; t < NT; t++)
                *reinterpret_cast<double2*>(dst + (8 * mt + lr) * LP + 8 * t + 2 * lc) =
                    make_double2(((acc[0][t][0] + acc[1][t][0]) + acc[2][t][0]) + acc[3][t][0],
                                 ((acc[0][t][1] + acc[1][t][1]) + acc[2][t][1]) + acc[3][t][1]);
        }
        __syncthreads();
        if (warp < 8) {  // Y <- T Y (T upper triangular: rows from the warp's own on)
            const double* T = T0 + (long long)b0 * ST_NB;
            double acc[NT][2];
#pragma unroll
            for (int t = 0; t < NT; t++) acc[t][0] = acc[t][1] = 0.0;
            for (int q = 8 * mt; q < ST_NB; q += 4) {
                double a = T[8 * mt + lr + (q + lc) * ST_NB];
                const int o = (q + lc) * LP + lr;
#pragma unroll
                for (int t = 0; t < NT; t++) dmma_8x8x4(acc[t][0], acc[t][1], a, ya[o + 8 * t] + yh[o + 8 * t]);
            }
#pragma unroll
            for (int t = 0; t < NT; t++)
                *reinterpret_cast<double2*>(yb + (8 * mt + lr) * LP + 8 * t + 2 * lc) = make_double2(acc[t][0], acc[t][1]);
        }
        __syncthreads();
        // Z -= V Y: eight rows at a time per warp, the next eight rows of V in flight
        double a[16];
        auto fetch = [&](int r0) {
            const int r = r0 + lr;
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const int c = 4 * q + lc;
                a[q] = c < jb && r < n ? V[r + (long long)(b0 + c) * n] : 0.0;
            }
        };
        fetch(b0 + 8 * warp);
        for (int r0 = b0 + 8 * warp; r0 < n; r0 += 8 * NW) {
            double av[16];
#pragma unroll
            for (int q = 0; q < 16; q++) av[q] = a[q];
            fetch(r0 + 8 * NW);
            double acc[NT][2];
#pragma unroll
            for (int t = 0; t < NT; t++) acc[t][0] = acc[t][1] = 0.0;
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const double* yr = yb + (4 * q + lc) * LP + lr;
#pragma unroll
                for (int t = 0; t < NT; t++) dmma_8x8x4(acc[t][0], acc[t][1], av[q], yr[8 * t]);
            }
            double* zr = z + (r0 + lr) * LP + 2 * lc;
#pragma unroll
            for (int t = 0; t < NT; t++) {
                double2 v = *reinterpret_cast<double2*>(zr + 8 * t);
                v.x -= acc[t][0];
                v.y -= acc[t][1];
                *reinterpret_cast<double2*>(zr + 8 * t) = v;
            }
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < n * NC; e += blockDim.x) {
        int r = e % n, c = e / n;
        if (c0 + c < k) S.Z[mat + r + (long long)(c0 + c) * n] = z[r * LP + c];
    }
    stage_stop<PROF>(S, m, 5);
}

}  // namespace axg
