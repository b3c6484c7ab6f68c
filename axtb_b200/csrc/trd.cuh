// Householder tridiagonalisation with the matrix on chip: one molecule per thread-block cluster
// (k_trd) or on the whole cooperative grid (k_trd_grid), its columns spread cyclically over the
// CTAs and kept in registers (the rest of a CTA's columns in its shared memory) from the first
// reflector to the last.
//
// The blocked reduction of the team kernel (team_tridiag_blocked) reads the trailing matrix from
// L2 once per column and carries the panel's pending reflectors through every row: per column a
// chain of load rounds and five barriers. Here the pass over the trailing matrix that multiplies
// it with the new reflector also applies the previous one (A -= v w^T + w v^T, then y = A v', both
// on the element while it is in a register: no panels, no dot products with them, no trailing
// GEMMs), and the full matrix is stored, so a column's product is complete inside the warp that
// owns the column: the CTAs exchange only y (each CTA its columns' entries) and the next column,
// behind ONE barrier per reflector. Everything of size n (w, the next column brought up to date,
// its norm, the next reflector) is then formed by every CTA for itself, with the same bits.
//
// Thread layout of a CTA (256 threads): warp = (row group rg of AW, column group cg of TC = 8/AW).
// Row (k AW + rg) 32 + lane is the thread's row slot k < RT; the CTA's local column l (global
// column l G + rank) belongs to column group l % TC, slot l / TC: slots below CR in registers
// (RT x CR values per thread), the others in shared memory. Rows and columns die from the front,
// so the row slots and column slots below the first live one are skipped. A column's dot product
// runs over the thread's rows in order, then over the lanes by a butterfly, then (AW > 1) over the
// row groups in order: its bits depend on n only, not on the number of CTAs.
#pragma once
#include <cfloat>
#include <type_traits>

#include "team_la.cuh"

namespace axg {

constexpr int TRD_THREADS = 256;
constexpr int TRD_SMEM_MAX = 227 * 1024;

// shared memory of one CTA (doubles): v (two buffers), w, the published column and y entries (two
// buffers each, cluster only), reduction slots, the row groups' partial y (grid only), columns
__host__ __device__ constexpr int trd_stride(int n) { return (n + 31) & ~31; }
__host__ __device__ constexpr int trd_slots(int n, int G, int TC) { return ((n + G - 1) / G + TC - 1) / TC; }
__host__ __device__ constexpr int trd_smem_cols(int n, int G, int TC, int CR) {
    return trd_slots(n, G, TC) > CR ? (trd_slots(n, G, TC) - CR) * TC : 0;
}
__host__ __device__ constexpr int trd_ylen(int n, int G, int TC) { return trd_slots(n, G, TC) * TC; }
__host__ __device__ constexpr long long trd_smem_doubles(int n, int G, int AW, int CR, bool grid) {
    return (long long)trd_stride(n) * (grid ? 3 : 5) + 48 + (grid ? AW : 2) * trd_ylen(n, G, 8 / AW) +
           (long long)trd_smem_cols(n, G, 8 / AW, CR) * trd_stride(n);
}

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ double ld_cluster(unsigned a) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void trd_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// sums over the warp of four values per lane: the sum of value 2 b4 + b3 (b_k = bit k of the lane)
__device__ __forceinline__ double warp_sum4(double y0, double y1, double y2, double y3) {
    int lane = threadIdx.x & 31;
    bool h = (lane & 16) != 0;
    double a = (h ? y2 : y0) + __shfl_xor_sync(0xffffffffu, h ? y0 : y2, 16);
    double b = (h ? y3 : y1) + __shfl_xor_sync(0xffffffffu, h ? y1 : y3, 16);
    h = (lane & 8) != 0;
    double s = (h ? b : a) + __shfl_xor_sync(0xffffffffu, h ? a : b, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}

// One molecule: A = F (n x n, column-major, lower triangle valid) -> d, e, tau, and the reflectors
// v_j over column j of F (zeros down to row j, one at row j + 1). xpub (grid only): 4 n doubles of
// global memory for the published column and y.
template <int RT, int CR, int AW, bool GRID>
__device__ __forceinline__ void trd_mol(int rank, int G, int n, double* __restrict__ F, double* __restrict__ d,
                                        double* __restrict__ e, double* __restrict__ tau, double* xpub) {
    constexpr int TC = 8 / AW;
    constexpr int EQ = (32 * AW * RT + TRD_THREADS - 1) / TRD_THREADS;  // vector elements per thread
    constexpr int EB = EQ < 5 ? EQ : 5;                                  // ... in flight at a time
    static_assert(GRID || EQ == EB, "cluster classes read a thread's elements in one go");
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int rg = wid % AW, cg = wid / AW;
    const int ns = trd_stride(n), ylen = trd_ylen(n, G, TC);
    const int nslot = trd_slots(n, G, TC);
    double* sv = s_work;              // two buffers
    double* sw = sv + 2 * ns;
    double* sred = sw + ns;           // 2 x 8 partials, alpha
    double* spub = sred + 48;         // cluster: y (2 x ylen) and column (2 x ns); grid: partial y (AW x ylen)
    double* scol = GRID ? spub + AW * ylen : spub + 2 * ylen + 2 * ns;
    auto col_of = [&](int slot) { return (slot * TC + cg) * G + rank; };
    auto row_of = [&](int k) { return (k * AW + rg) * 32 + lane; };
    auto elem = [&](int r, int c) {
        return (r < n && c < n) ? (r >= c ? F[r + (long long)c * n] : F[c + (long long)r * n]) : 0.0;
    };
    // ---- the CTA's columns
    double A[RT][CR];
#pragma unroll
    for (int s = 0; s < CR; s++) {
        const int c = col_of(s);
#pragma unroll
        for (int k = 0; k < RT; k++) A[k][s] = elem(row_of(k), c);
    }
    for (int s = CR; s < nslot; s++) {
        const int c = col_of(s);
        double* p = scol + (long long)((s - CR) * TC + cg) * ns;
        for (int k = 0; k < RT; k++)
            if ((k * AW + rg) * 32 < ns) p[row_of(k)] = elem(row_of(k), c);
    }
    for (int i = tid; i < 3 * ns; i += TRD_THREADS) sv[i] = 0.0;
    // publish column jn (held in register slot s of this warp's column group)
    auto pub_reg = [&](double* dst, int s) {
#pragma unroll
        for (int u = 0; u < CR; u++)
            if (u == s) {
#pragma unroll
                for (int k = 0; k < RT; k++)
                    if ((k * AW + rg) * 32 < ns) {
                        if (GRID) {
                            if (row_of(k) < n) __stcg(dst + row_of(k), A[k][u]);
                        } else dst[row_of(k)] = A[k][u];
                    }
            }
    };
    auto pub_col = [&](int par) { return GRID ? xpub + par * n : spub + 2 * ylen + par * ns; };
    if (rank == 0 && cg == 0) pub_reg(pub_col(0), 0);
    auto barrier = [&]() {
        if (GRID) cg::this_grid().sync();
        else trd_cluster_sync();
    };
    barrier();  // column 0 is published (and every CTA has read F: the reflectors go over it)
    // cluster addresses of this thread's y entries (buffer 0)
    unsigned yaddr[EQ];
    if (!GRID) {
#pragma unroll
        for (int q = 0; q < EQ; q++) {
            int i = tid + q * TRD_THREADS;
            yaddr[q] = cluster_addr(smem_addr(spub) + 8 * (i / G), i % G);
        }
    }
    int cur = 0, own = 0, jl = 0;  // column j: CTA own, local column jl
    double tj = 0.0;
    for (int j = 0;; j++) {
        const int par = j & 1;
        double* v = sv + cur * ns;
        double* vn = sv + (cur ^ 1) * ns;
        // (1) the published column j and y; y . v
        unsigned ca = 0;
        double yj;
        if (GRID) {
            yj = j > 0 ? __ldcg(xpub + 2 * n + par * n + j) : 0.0;
        } else {
            ca = cluster_addr(smem_addr(pub_col(par)), own);
            yj = j > 0 ? ld_cluster(cluster_addr(smem_addr(spub + par * ylen) + 8 * jl, own)) : 0.0;
        }
        double dot = 0.0;
#pragma unroll
        for (int q0 = 0; q0 < EQ; q0 += EB) {
            double cv[EB], yv[EB];
#pragma unroll
            for (int q = 0; q < EB; q++) {
                int i = tid + (q0 + q) * TRD_THREADS;
                bool ok = q0 + q < EQ && i >= j && i < n;
                if (GRID) {
                    cv[q] = ok ? __ldcg(xpub + par * n + i) : 0.0;
                    yv[q] = ok && j > 0 ? __ldcg(xpub + 2 * n + par * n + i) : 0.0;
                } else {
                    cv[q] = ok ? ld_cluster(ca + 8 * i) : 0.0;
                    yv[q] = ok && j > 0 ? ld_cluster(yaddr[q] + 8 * par * ylen) : 0.0;
                }
            }
#pragma unroll
            for (int q = 0; q < EB; q++) {
                int i = tid + (q0 + q) * TRD_THREADS;
                if (q0 + q < EQ && i < ns) {
                    dot = fma(yv[q], v[i], dot);
                    vn[i] = cv[q];
                    sw[i] = yv[q];
                }
            }
        }
        dot = warp_sum(dot);
        if (lane == 0) sred[wid] = dot;
        __syncthreads();
        double ds = 0.0;
#pragma unroll
        for (int q = 0; q < 8; q++) ds += sred[q];
        // (2) w = tau (y - tau/2 (y.v) v); column j brought up to date with the previous reflector
        const double kap = 0.5 * tj * ds;
        const double vj = v[j], wj = tj * (yj - kap * vj);
        double xs = 0.0;
#pragma unroll
        for (int q = 0; q < EQ; q++) {
            int i = tid + q * TRD_THREADS;
            if (i < ns && i >= j) {
                double vi = v[i], w = tj * (sw[i] - kap * vi);
                double a = vn[i] - vi * wj - w * vj;
                sw[i] = w;
                vn[i] = a;
                if (i == j && rank == 0) d[j] = a;
                if (i == j + 1) sred[16] = a;
                if (i > j + 1) xs = fma(a, a, xs);
            }
        }
        xs = warp_sum(xs);
        if (lane == 0) sred[8 + wid] = xs;
        __syncthreads();
        const double alpha = sred[16];
        if (j == n - 2) {  // the last 2 x 2 block: its lower right element takes the last reflector
            if (tid == 0 && rank == 0) {
                e[j] = alpha;
                tau[j] = 0.0;
                e[n - 1] = 0.0;
                tau[n - 1] = 0.0;
            }
            const int c = n - 1;
            auto last = [&](double a) { d[n - 1] = a - v[c] * sw[c] - sw[c] * v[c]; };
#pragma unroll
            for (int s = 0; s < CR; s++)
#pragma unroll
                for (int k = 0; k < RT; k++)
                    if (col_of(s) == c && row_of(k) == c) last(A[k][s]);
            for (int s = CR; s < nslot; s++)
                if (col_of(s) == c && (c >> 5) % AW == rg && (c & 31) == lane)
                    last(scol[(long long)((s - CR) * TC + cg) * ns + c]);
            break;
        }
        double xn2 = 0.0;
#pragma unroll
        for (int q = 0; q < 8; q++) xn2 += sred[8 + q];
        // (3) the Householder vector of column j
        double beta, scale;
        if (xn2 == 0.0) {
            tj = 0.0;
            beta = alpha;
            scale = 0.0;
        } else {
            beta = -copysign(sqrt(alpha * alpha + xn2), alpha);
            tj = (beta - alpha) / beta;
            scale = 1.0 / (alpha - beta);
        }
        if (tid == 0 && rank == 0) {
            e[j] = beta;
            tau[j] = tj;
        }
#pragma unroll
        for (int q = 0; q < EQ; q++) {
            int i = tid + q * TRD_THREADS;
            if (i < ns) {
                double x = i > j + 1 ? vn[i] * scale : (i == j + 1 ? 1.0 : 0.0);
                vn[i] = x;
                if (i <= j) sw[i] = 0.0;
                if (rank == own && i < n) F[i + (long long)j * n] = x;
            }
        }
        __syncthreads();
        // (4) the pass: previous reflector applied, product with the new one
        const int jn = j + 1, npar = par ^ 1;
        double* cdst = pub_col(npar);
        auto put = [&](int slot, double y0, double y1, double y2, double y3, int cnt) {
            double s = warp_sum4(y0, y1, y2, y3);
            int u = ((lane >> 4) & 1) * 2 + ((lane >> 3) & 1);
            if ((lane & 7) == 0 && u < cnt) {
                int l = (slot + u) * TC + cg;
                if (AW > 1) spub[rg * ylen + l] = s;
                else if (GRID) {
                    if (l * G + rank < n) __stcg(xpub + 2 * n + npar * n + l * G + rank, s);
                } else spub[npar * ylen + l] = s;
            }
        };
#pragma unroll
        for (int g = 0; g < CR; g += 4) {
            constexpr int GS = 4;
            // skipped: no columns of this molecule, or all of them done
            if (g >= nslot || col_of(g + 3 < CR ? g + 3 : CR - 1) < jn) continue;
            double wc[GS], vc[GS], y[GS];
#pragma unroll
            for (int u = 0; u < GS; u++) {
                int c = col_of(g + u);
                bool ok = g + u < CR && c < n;
                wc[u] = ok ? sw[c] : 0.0;
                vc[u] = ok ? v[c] : 0.0;
                y[u] = 0.0;
            }
#pragma unroll
            for (int k = 0; k < RT; k++) {
                const int b = (k * AW + rg) * 32;
                if (b + 31 >= jn && b < ns) {
                    double vr = v[b + lane], wr = sw[b + lane], nr = vn[b + lane];
#pragma unroll
                    for (int u = 0; u < GS; u++)
                        if (g + u < CR) {
                            double a = A[k][g + u];
                            a = fma(-vr, wc[u], a);
                            a = fma(-wr, vc[u], a);
                            A[k][g + u] = a;
                            y[u] = fma(a, nr, y[u]);
                        }
                }
            }
#pragma unroll
            for (int u = 0; u < GS; u++)
                if (g + u < CR && col_of(g + u) == jn) pub_reg(cdst, g + u);
            put(g, y[0], y[1], y[2], y[3], min(g + 4 <= CR ? 4 : CR - g, nslot - g));
        }
        const int k0 = jn / (32 * AW);  // row slots below hold finished rows only
        for (int s = CR; s < nslot; s += 4) {
            const int cnt = min(4, nslot - s);
            if (col_of(s + cnt - 1) < jn) continue;
            double wc[4], vc[4], y[4];
            double* p = scol + (long long)((s - CR) * TC + cg) * ns;
            const long long cs = (long long)TC * ns;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                int c = col_of(s + u);
                bool ok = u < cnt && c < n;
                wc[u] = ok ? sw[c] : 0.0;
                vc[u] = ok ? v[c] : 0.0;
                y[u] = 0.0;
            }
            auto rows = [&](auto CN) {
                constexpr int N = decltype(CN)::value;
#pragma unroll 2
                for (int k = k0; k < RT; k++) {
                    const int b = (k * AW + rg) * 32;
                    if (b >= ns) break;
                    const int r = b + lane;
                    double vr = v[r], wr = sw[r], nr = vn[r], a[N];
#pragma unroll
                    for (int u = 0; u < N; u++) a[u] = p[u * cs + r];
#pragma unroll
                    for (int u = 0; u < N; u++) {
                        a[u] = fma(-vr, wc[u], a[u]);
                        a[u] = fma(-wr, vc[u], a[u]);
                        p[u * cs + r] = a[u];
                        y[u] = fma(a[u], nr, y[u]);
                    }
                }
            };
            if (cnt == 4) rows(std::integral_constant<int, 4>());
            else if (cnt == 3) rows(std::integral_constant<int, 3>());
            else if (cnt == 2) rows(std::integral_constant<int, 2>());
            else rows(std::integral_constant<int, 1>());
            for (int u = 0; u < cnt; u++)
                if (col_of(s + u) == jn) {
                    for (int k = 0; k < RT; k++) {
                        const int b = (k * AW + rg) * 32;
                        if (b >= ns) break;
                        double a = p[u * cs + b + lane];
                        if (GRID) {
                            if (b + lane < n) __stcg(cdst + b + lane, a);
                        } else cdst[b + lane] = a;
                    }
                }
            put(s, y[0], y[1], y[2], y[3], cnt);
        }
        if (AW > 1) {
            __syncthreads();
            for (int l = tid; l < ylen; l += TRD_THREADS) {
                int c = l * G + rank;
                if (c >= jn && c < n) {
                    double s = spub[l];
#pragma unroll
                    for (int q = 1; q < AW; q++) s += spub[q * ylen + l];
                    __stcg(xpub + 2 * n + npar * n + c, s);
                }
            }
        }
        barrier();
        cur ^= 1;
        if (++own == G) {
            own = 0;
            jl++;
        }
    }
    barrier();  // no CTA leaves (or starts the next molecule) while another reads its memory
}

// SM cycles of the reduction into the profiler's counters (the molecule's counter in units of the
// team kernel's half-SM CTAs)
__device__ __forceinline__ void trd_cycles(const State& S, int m, int rank, int G, long long t0) {
    if (rank == 0 && threadIdx.x == 0) {
        double c = 2.0 * G * (double)(clock64() - t0);
        S.mol_cyc[m] += c;
        atomicAdd(&g_team_cycles[1], (unsigned long long)c);
    }
}

// One cluster per molecule of `list` (one-CTA-team molecules of the batch), CTAs of a cluster by
// their rank. Launched per size class with the class's row slots and cluster size.
template <int RT, int CR>
__global__ void __launch_bounds__(TRD_THREADS, 1) k_trd(Batch B, State S, const int* list, int cycles) {
    const long long t0 = clock64();
    unsigned rank, G;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(G));
    const int m = list[blockIdx.x / G];
    if (!S.active[m]) return;  // the same for the whole cluster
    const int n = B.m_nao[m], ao0 = B.m_ao0[m];
    trd_mol<RT, CR, 1, false>((int)rank, (int)G, n, S.Fp + B.m_mat0[m], S.dtri + ao0, S.etri + ao0, S.tau + ao0, nullptr);
    if (cycles) trd_cycles(S, m, (int)rank, (int)G, t0);
}

// One molecule on the whole cooperative grid; xpub: 4 n doubles
template <int RT, int CR>
__global__ void __launch_bounds__(TRD_THREADS, 1) k_trd_grid(Batch B, State S, int m, double* xpub, int cycles) {
    const long long t0 = clock64();
    if (!S.active[m]) return;  // uniform over the grid
    const int n = B.m_nao[m], ao0 = B.m_ao0[m];
    trd_mol<RT, CR, 8, true>((int)blockIdx.x, (int)gridDim.x, n, S.Fp + B.m_mat0[m], S.dtri + ao0, S.etri + ao0, S.tau + ao0,
                             xpub);
    if (cycles) trd_cycles(S, m, (int)blockIdx.x, (int)gridDim.x, t0);
}

// ---- size classes
struct TrdClass {
    int rt, cr;
    const void* fn;
};
// cluster path: row slots per thread (n <= 32 rt) and register columns per warp
inline const TrdClass* trd_classes(int& count) {
    static const TrdClass c[] = {{4, 16, (const void*)k_trd<4, 16>}, {6, 12, (const void*)k_trd<6, 12>},
                                 {8, 9, (const void*)k_trd<8, 9>},   {12, 6, (const void*)k_trd<12, 6>},
                                 {16, 5, (const void*)k_trd<16, 5>}, {19, 4, (const void*)k_trd<19, 4>},
                                 {24, 3, (const void*)k_trd<24, 3>}};
    count = 7;
    return c;
}
// whole grid: n <= 256 rt, columns per CTA in registers
inline const TrdClass* trd_grid_classes(int& count) {
    static const TrdClass c[] = {{4, 8, (const void*)k_trd_grid<4, 8>},   {5, 9, (const void*)k_trd_grid<5, 9>},
                                 {6, 11, (const void*)k_trd_grid<6, 11>}, {7, 12, (const void*)k_trd_grid<7, 12>},
                                 {8, 10, (const void*)k_trd_grid<8, 10>}, {10, 8, (const void*)k_trd_grid<10, 8>}};
    count = 6;
    return c;
}

}  // namespace axg
