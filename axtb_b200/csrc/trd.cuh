// Householder tridiagonalisation with the matrix on chip: one molecule per thread-block cluster
// (k_trd) or on a cooperative grid or a team of it (k_trd_grid, k_trd_teams), its columns spread cyclically over the
// CTAs and kept in registers (the rest of a CTA's columns in its shared memory) from the first
// reflector to the last.
//
// The blocked reduction of the team kernel (team_tridiag_blocked) reads the trailing matrix from
// L2 once per column and carries the panel's pending reflectors through every row: per column a
// chain of load rounds and five barriers. Here the pass over the trailing matrix that multiplies
// it with the new reflector also applies the previous one (A -= v w^T + w v^T, then y = A v', both
// on the element while it is in a register: no panels, no dot products with them, no trailing
// GEMMs), and the full matrix is stored, so a column's product is complete inside the warp that
// owns the column: the CTAs exchange only y and the next column (as the next row: each CTA its own
// columns' two entries, so that no CTA serves a whole column to all the others). In a cluster every
// warp pushes its columns' pairs into each CTA's shared memory as soon as it has them (st.async; a
// transaction barrier counts the bytes), so one one-way trip is all that separates two reflectors;
// the grid's pairs go through global memory, each with its own flag. Everything of size n (w, the next column brought up to date,
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
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"
#include "trd_classes.h"

namespace axg {
namespace cg = cooperative_groups;

extern __shared__ __align__(16) double s_trd[];

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void trd_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a pair into another CTA's shared memory; its barrier there counts the bytes
__device__ __forceinline__ void push_pair(unsigned dst, unsigned bar, double x, double y) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "d"(x), "d"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// waits (at most ~2^22 tries) for the barrier's phase to complete; false when it gave up
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned phase) {
    for (int it = 0; it < (1 << 22); it++) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(phase)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// The grid's pairs (row element, y entry) travel through global memory as single 128-bit words that
// carry their own flag: the values are scaled by 2^-500 (|x| < 2^500; exact from 2^-522 up, and what is
// below loses bits that no sum with the matrix's other elements holds), which leaves the
// top exponent bit of the row element zero and free for the phase of the buffer's use. A reader
// checks the very words it needs, so no fence has to order them: a count of the CTAs that have
// published tells one thread per CTA when to look (all threads polling their words from the start
// kept L2 busy: 7.4 us per reflector at 1202 rows instead of 3.8 behind a grid barrier).
__device__ __forceinline__ void st_pair(double* p, double x, double y, unsigned phase, int* status) {
    const double big = 3.273390607896142e150, down = 3.054936363499605e-151;  // 2^500, 2^-500
    if (!(fabs(x) < big) || !(fabs(y) < big)) {
        atomicOr(status, ST_NONFINITE);
        x = y = 0.0;
    }
    const long long a = __double_as_longlong(x * down) | (long long)phase << 62, b = __double_as_longlong(y * down);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p), "l"(a),
                 "l"(b)
                 : "memory");
}
__device__ __forceinline__ void ld_pair(const double* p, long long& a, long long& b) {
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ bool pair_ready(long long a, unsigned phase) { return (unsigned)(a >> 62 & 1) == phase; }
__device__ __forceinline__ double2 unpack_pair(long long a, long long b) {
    const double up = 3.273390607896142e150;
    return make_double2(__longlong_as_double(a & ~(1LL << 62)) * up, __longlong_as_double(b) * up);
}
// a shared-memory load the compiler keeps where it is written (ahead of the branch that uses it)
__device__ __forceinline__ double lds_now(unsigned a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
// sum of the eight warps' partials, in a fixed order
__device__ __forceinline__ double sum8(const double* p) {
    return ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
}

// sums over the warp of N values per lane (N = 1, 2, 4 or 8), each lane ending with the sum of one:
// value `warp_sum_slot<N>(lane)`, the same tree for every value
template <int N>
__device__ __forceinline__ double warp_sum_n(const double* y) {
    double t[N];
#pragma unroll
    for (int u = 0; u < N; u++) t[u] = y[u];
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int w = N / 2; w >= 1; w >>= 1, o >>= 1) {
        const bool h = (lane & o) != 0;
#pragma unroll
        for (int u = 0; u < w; u++) {
            double keep = h ? t[w + u] : t[u], send = h ? t[u] : t[w + u];
            t[u] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (; o >= 1; o >>= 1) t[0] += __shfl_xor_sync(0xffffffffu, t[0], o);
    return t[0];
}
// the value a lane holds: its top log2(N) bits
template <int N>
__device__ __forceinline__ int warp_sum_slot(int lane) {
    return N == 8 ? lane >> 2 : N == 4 ? lane >> 3 : N == 2 ? lane >> 4 : 0;
}

// One molecule: A = F (n x n, column-major, lower triangle valid) -> d, e, tau, and the reflectors
// v_j over column j of F (zeros down to row j, one at row j + 1). xpub (grid only): 4 n doubles of
// global memory for the published pairs, and their count. false: a wait for the other CTAs gave up.
template <int RT, int CR, int AW, bool GRID>
__device__ __forceinline__ bool trd_mol(int rank, int G, int n, double* __restrict__ F, double* __restrict__ d,
                                        double* __restrict__ e, double* __restrict__ tau, double* xpub,
                                        int* status) {
    constexpr int TC = 8 / AW;
    constexpr int EQ = (32 * AW * RT + TRD_THREADS - 1) / TRD_THREADS;  // vector elements per thread
    constexpr int EB = EQ < 5 ? EQ : 5;                                  // ... in flight at a time
    constexpr int GS = CR <= 8 ? CR : (CR + 1) / 2;  // register columns taken at a time
    constexpr int NSUM = CR <= 4 ? 4 : 8, CY = (CR + NSUM - 1) / NSUM * NSUM;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int rg = wid % AW, cg = wid / AW;
    const int ns = trd_stride(n), ylen = trd_ylen(n, G, TC);
    const int nslot = trd_slots(n, G, TC);
    double* sv = s_trd;              // two buffers
    double* sw = sv + 2 * ns;
    double* sred = sw + ns;           // 2 x 8 partials, alpha; two barriers
    double* rcv = sred + 48;          // cluster: received pairs (two buffers of ns)
    double* stg = rcv + (GRID ? 0 : 4 * ns);  // cluster: own pairs; grid: partial y (AW x ylen)
    double* spiv = stg + (GRID ? AW : 2) * ylen;  // register columns: the rows of the next row's block of 32
    double* srow = spiv + 32 * CR * TC;  // grid: the next row's elements
    double* scol = srow + (GRID ? ylen : 0);
    const unsigned bar0 = smem_addr(sred + 24);
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
    if (!GRID && tid == 0) {
        bar_init(bar0);
        bar_init(bar0 + 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        bar_expect(bar0, 16 * n);
    }
    if (!GRID) {
        __syncthreads();
        trd_cluster_sync();  // the barriers are ready (and every CTA has read F: the reflectors go over it)
    }
    // element (next row, column of `slot`) of the CTA's own pairs
    auto put_row = [&](int slot, double a) {
        const int l = slot * TC + cg;
        if (GRID) srow[l] = a;
        else stg[2 * l] = a;
    };
    // this lane's part of the pairs' distribution: CTA lane % G, slots lane / G, + 32 / G, ...
    const int per = GRID ? 1 : 32 / G, dslot = GRID ? 0 : lane / G;
    unsigned drcv = 0, dbar = 0;
    if (!GRID) {
        drcv = cluster_addr(smem_addr(rcv), lane % G);
        dbar = cluster_addr(bar0, lane % G);
    }
    auto push = [&](int par, int first) {  // the warp's live columns (from column `first` on) to every CTA
        if (GRID) return;
        __syncwarp();
        if (dslot < per)
            for (int s = dslot; s < nslot; s += per) {
                const int l = s * TC + cg, c = l * G + rank;
                if (c >= first && c < n) {
                    double2 v = reinterpret_cast<const double2*>(stg)[l];
                    push_pair(drcv + 16 * (par * ns + c), dbar + 8 * par, v.x, v.y);
                }
            }
        __syncwarp();
    };
    // The block of 32 rows that holds the next row lives in shared memory (one value per lane and
    // register column): the register code then needs no row picked by a run-time index.
    double* pv = spiv + 32 * cg + lane;
    auto to_pivot = [&](int kb) {  // row slot kb of this thread
#pragma unroll
        for (int k = 0; k < RT; k++)
            if (k == kb) {
#pragma unroll
                for (int s = 0; s < CR; s++) pv[32 * TC * s] = A[k][s];
            }
    };
    // row 0 (= column 0) is published first
    if (rg == 0) {
        to_pivot(0);
        if (lane == 0) {
            for (int s = 0; s < nslot; s++)
                put_row(s, s < CR ? pv[32 * TC * s] : scol[(long long)((s - CR) * TC + cg) * ns]);
            if (!GRID)
                for (int s = 0; s < nslot; s++) stg[2 * (s * TC + cg) + 1] = 0.0;
        }
    }
    push(0, 0);
    bool ok = true;
    unsigned* gate = reinterpret_cast<unsigned*>(xpub + 4 * (long long)n);
    // grid: the CTA's pairs from column `first` on, the row groups' products summed in order
    auto publish = [&](int par, int first, unsigned phase, bool products) {
        __syncthreads();
        for (int l = tid; l < ylen; l += TRD_THREADS) {
            int c = l * G + rank;
            if (c >= first && c < n) {
                double s = 0.0;
                if (products) {
                    s = stg[l];
#pragma unroll
                    for (int q = 1; q < AW; q++) s += stg[q * ylen + l];
                }
                st_pair(xpub + 2 * ((long long)par * n + c), srow[l], s, phase, status);
            }
        }
        // the count only says when to look (other warps' pairs may still be on their way): the words' flags decide
        if (tid < 32) {
            __syncwarp();
            if (tid == 0) asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(gate) : "memory");
        }
    };
    if (GRID) {
        publish(0, 0, 1, false);
        cg::this_grid().sync();  // every CTA has read F: the reflectors go over it
    }
    int cur = 0, own = 0;  // own: the CTA that stores reflector j
    double tj = 0.0;
    for (int j = 0;; j++) {
        const int par = j & 1;
        double* v = sv + cur * ns;
        double* vn = sv + (cur ^ 1) * ns;
        // (1) the published row j and y; y . v
        const int j0 = min(j, n - G);  // every CTA publishes at least one pair, live or not: none runs two ahead
        const unsigned phase = (j >> 1 & 1) ^ 1;
        const double2* prow = reinterpret_cast<const double2*>(rcv) + par * ns;
        if (!GRID) {
            // every pair has arrived: every warp with live columns, this CTA's too, has finished its
            // last pass, and every CTA has read the buffer that the next pairs go to
            if (ok) ok = bar_wait(bar0 + 8 * par, (j >> 1) & 1);
            if (tid == 0 && j + 2 < n) bar_expect(bar0 + 8 * (par ^ 1), 16 * (n - min(j + 1, n - G)));
        }
        if (GRID) {  // one thread watches the count of CTAs that have published; the words' flags decide
            if (tid == 0) {
                const unsigned want = (unsigned)G * (j + 1);
                unsigned c = 0;
                for (int it = 0; ok && c < want && it < (1 << 22); it++)
                    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(gate) : "memory");
            }
            __syncthreads();
        }
        double dot = 0.0;
#pragma unroll
        for (int q0 = 0; q0 < EQ; q0 += EB) {
            double2 pv[EB];
            if (GRID) {
                long long pa[EB], pb[EB];
                bool in = false;
                for (int it = 0; !in && it < (1 << 20); it++) {
                    in = true;
#pragma unroll
                    for (int q = 0; q < EB; q++) {
                        int i = tid + (q0 + q) * TRD_THREADS;
                        if (q0 + q < EQ && i >= j0 && i < n)
                            ld_pair(xpub + 2 * ((long long)par * n + i), pa[q], pb[q]);
                        else pa[q] = (long long)phase << 62, pb[q] = 0;
                    }
#pragma unroll
                    for (int q = 0; q < EB; q++) in = in && pair_ready(pa[q], phase);
                    if (!ok) break;
                }
                ok = ok && in;
#pragma unroll
                for (int q = 0; q < EB; q++) pv[q] = unpack_pair(pa[q], pb[q]);
            } else {
#pragma unroll
                for (int q = 0; q < EB; q++) {
                    int i = tid + (q0 + q) * TRD_THREADS;
                    pv[q] = make_double2(0.0, 0.0);
                    if (q0 + q < EQ && i >= j && i < n) pv[q] = prow[i];
                }
            }
#pragma unroll
            for (int q = 0; q < EB; q++) {
                int i = tid + (q0 + q) * TRD_THREADS;
                if (q0 + q < EQ && i < ns) {
                    if (i < j) pv[q] = make_double2(0.0, 0.0);
                    dot = fma(pv[q].y, v[i], dot);
                    vn[i] = pv[q].x;
                    sw[i] = pv[q].y;
                    if (i == j) sred[17] = pv[q].y;
                }
            }
        }
        dot = warp_sum(dot);
        if (lane == 0) sred[wid] = dot;
        __syncthreads();
        const double ds = sum8(sred);
        // (2) w = tau (y - tau/2 (y.v) v); column j brought up to date with the previous reflector
        const double kap = 0.5 * tj * ds;
        const double vj = v[j], wj = tj * (sred[17] - kap * vj);
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
            const bool here = (c >> 5) % AW == rg && (c & 31) == lane;
            if ((c & 31) == 0 && here) to_pivot(c / (32 * AW));  // a row block of its own, not reached before
            for (int s = 0; s < nslot; s++)
                if (col_of(s) == c && here)
                    last(s < CR ? pv[32 * TC * s] : scol[(long long)((s - CR) * TC + cg) * ns + c]);
            break;
        }
        const double xn2 = sum8(sred + 8);
        // (3) the Householder vector of column j
        double beta, scale;
        if (xn2 == 0.0) {
            tj = 0.0;
            beta = alpha;
            scale = 0.0;
        } else {
            // one reciprocal square root for both roots' uses: |beta| = sqrt(ss) after a Newton
            // correction, tau = (beta - alpha) / beta = 1 + |alpha| / |beta|
            const double ss = fma(alpha, alpha, xn2), r = rsqrt(ss), b0 = ss * r;
            const double ab = fma(0.5 * r, fma(-b0, b0, ss), b0);
            beta = -copysign(ab, alpha);
            tj = fma(fabs(alpha), r, 1.0);
            scale = 1.0 / (alpha - beta);
        }
        if (tid == 0 && rank == 0) {
            e[j] = beta;
            tau[j] = tj;
        }
        const bool mine = rank == own;
        if (++own == G) own = 0;
#pragma unroll
        for (int q = 0; q < EQ; q++) {
            int i = tid + q * TRD_THREADS;
            if (i < ns) {
                double x = i > j + 1 ? vn[i] * scale : (i == j + 1 ? 1.0 : 0.0);
                vn[i] = x;
                if (i <= j) sw[i] = 0.0;
                if (mine && i < n) F[i + (long long)j * n] = x;
            }
        }
        __syncthreads();
        // (4) the pass: previous reflector applied, product with the new one
        const int jn = j + 1, npar = par ^ 1;
        auto put = [&](int slot, double s) {  // the product of column `slot`, its sum in this lane
            const int l = slot * TC + cg;
            if (GRID) stg[rg * ylen + l] = s;
            else stg[2 * l + 1] = s;
        };
        const unsigned av = smem_addr(v + rg * 32 + lane), aw = smem_addr(sw + rg * 32 + lane),
                       an = smem_addr(vn + rg * 32 + lane);
        const bool has_row = (jn >> 5) % AW == rg;  // this row group has the next row
        const int kb = jn / (32 * AW);
        if ((jn & 31) == 0 && has_row) to_pivot(kb);
        const int b1 = AW == 1 ? 32 * RT : ns;  // AW = 1: RT is n's own, no row slot is empty
        double y[CY];
#pragma unroll
        for (int u = 0; u < CY; u++) y[u] = 0.0;
#pragma unroll
        for (int g = 0; g < CR; g += GS) {
            // skipped: no columns of this molecule, or all of them done
            if (g >= nslot || col_of(g + GS - 1 < CR ? g + GS - 1 : CR - 1) < jn) continue;
            double wc[GS], vc[GS];
#pragma unroll
            for (int u = 0; u < GS; u++) {
                int c = min(col_of(g + u), n - 1);  // a column the molecule does not have: never pushed
                wc[u] = sw[c];
                vc[u] = v[c];
            }
            double vr = lds_now(av), wr = lds_now(aw), nr = lds_now(an);
            if (has_row) {
                const double v0 = lds_now(av + 256 * AW * kb), w0 = lds_now(aw + 256 * AW * kb),
                             n0 = lds_now(an + 256 * AW * kb);
                double a[GS];
#pragma unroll
                for (int u = 0; u < GS; u++)
                    if (g + u < CR) a[u] = pv[32 * TC * (g + u)];
#pragma unroll
                for (int u = 0; u < GS; u++)
                    if (g + u < CR) {
                        a[u] = fma(-v0, wc[u], a[u]);
                        a[u] = fma(-w0, vc[u], a[u]);
                        pv[32 * TC * (g + u)] = a[u];
                        y[g + u] = a[u] * n0;
                    }
                if (lane == (jn & 31)) {
#pragma unroll
                    for (int u = 0; u < GS; u++)
                        if (g + u < CR && g + u < nslot) put_row(g + u, a[u]);
                }
            }
#pragma unroll
            for (int k = 0; k < RT; k++) {
                const int b = (k * AW + rg) * 32;
                const double v0 = vr, w0 = wr, n0 = nr;
                if (k + 1 < RT && b + 32 * AW < b1) {  // the next row slot's vectors, in flight meanwhile
                    vr = lds_now(av + 256 * AW * (k + 1));
                    wr = lds_now(aw + 256 * AW * (k + 1));
                    nr = lds_now(an + 256 * AW * (k + 1));
                }
                if (b > jn && b < b1) {
#pragma unroll
                    for (int u = 0; u < GS; u++)
                        if (g + u < CR) {
                            double a = A[k][g + u];
                            a = fma(-v0, wc[u], a);
                            a = fma(-w0, vc[u], a);
                            A[k][g + u] = a;
                            y[g + u] = fma(a, n0, y[g + u]);
                        }
                }
            }
        }
#pragma unroll
        for (int g = 0; g < CR; g += NSUM) {
            if (g < nslot) {
                double s = warp_sum_n<NSUM>(y + g);
                const int u = warp_sum_slot<NSUM>(lane);
                if ((lane & (32 / NSUM - 1)) == 0 && g + u < min(CR, nslot)) put(g + u, s);
            }
        }
        const int k0 = jn / (32 * AW);  // row slots below hold finished rows only
        const int k1 = min(RT, (ns / 32 - rg + AW - 1) / AW);
        for (int s = CR; s < nslot; s += 4) {
            const int cnt = min(4, nslot - s);
            if (col_of(s + cnt - 1) < jn) continue;
            double wc[4], vc[4], ys[4];
            const unsigned ac = smem_addr(scol + (long long)((s - CR) * TC + cg) * ns + rg * 32 + lane);
            const unsigned cs = 8 * TC * ns;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                int c = min(col_of(s + u), n - 1);
                wc[u] = sw[c];
                vc[u] = v[c];
                ys[u] = 0.0;
            }
            auto rows = [&](auto CN) {
                constexpr int N = decltype(CN)::value;
                constexpr int KU = N == 1 ? 4 : N == 2 ? 3 : 2;  // rows loaded together
                auto step = [&](auto KN, unsigned o) {
                    constexpr int K = decltype(KN)::value;
                    double v0[K], w0[K], n0[K], a[K][N];
#pragma unroll
                    for (int k = 0; k < K; k++) {
                        v0[k] = lds_now(av + o + 256 * AW * k);
                        w0[k] = lds_now(aw + o + 256 * AW * k);
                        n0[k] = lds_now(an + o + 256 * AW * k);
#pragma unroll
                        for (int u = 0; u < N; u++) a[k][u] = lds_now(ac + u * cs + o + 256 * AW * k);
                    }
#pragma unroll
                    for (int k = 0; k < K; k++)
#pragma unroll
                        for (int u = 0; u < N; u++) {
                            double x = fma(-v0[k], wc[u], a[k][u]);
                            x = fma(-w0[k], vc[u], x);
                            asm volatile("st.shared.f64 [%0], %1;" ::"r"(ac + u * cs + o + 256 * AW * k), "d"(x));
                            ys[u] = fma(x, n0[k], ys[u]);
                        }
                };
                int k = k0;
                for (; k + KU <= k1; k += KU) step(std::integral_constant<int, KU>(), 256 * AW * k);
                for (; k < k1; k++) step(std::integral_constant<int, 1>(), 256 * AW * k);
                if ((jn >> 5) % AW == rg && lane == (jn & 31)) {
#pragma unroll
                    for (int u = 0; u < N; u++) put_row(s + u, lds_now(ac + u * cs + 8 * ((jn & ~31) - rg * 32)));
                }
            };
            if (cnt == 4) rows(std::integral_constant<int, 4>());
            else if (cnt == 3) rows(std::integral_constant<int, 3>());
            else if (cnt == 2) rows(std::integral_constant<int, 2>());
            else rows(std::integral_constant<int, 1>());
            const double sum = warp_sum_n<4>(ys);
            if ((lane & 7) == 0 && (lane >> 3) < cnt) put(s + (lane >> 3), sum);
        }
        if (GRID) {
            publish(npar, min(jn, n - G), (jn >> 1 & 1) ^ 1, true);
        } else push(npar, min(jn, n - G));
        cur ^= 1;
    }
    // no CTA leaves (or starts the next molecule) while another writes its memory
    if (!GRID) trd_cluster_sync();
    return ok;
}

// SM cycles of the reduction into the molecule's counter and the profiler's slot (nullptr: not profiling), in
// units of the team kernel's half-SM CTAs
__device__ __forceinline__ void trd_cycles(const State& S, int m, int rank, int G, long long t0, unsigned long long* slot) {
    if (rank == 0 && threadIdx.x == 0) {
        const double c = 2.0 * G * (double)(clock64() - t0);
        S.mol_cyc[m] += c;
        atomicAdd(slot, (unsigned long long)c);
    }
}

// One cluster per molecule of `list` (one-CTA-team molecules of the batch), CTAs of a cluster by
// their rank. Launched per size class with the class's row slots and cluster size.
template <int RT, int CR>
__global__ void __launch_bounds__(TRD_THREADS, 1) k_trd(Batch B, State S, const int* list, unsigned long long* cycles) {
    const long long t0 = clock64();
    unsigned rank, G;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(G));
    const int m = list[blockIdx.x / G];
    if (!S.active[m]) return;  // the same for the whole cluster
    const int n = B.m_nao[m], ao0 = B.m_ao0[m];
    if (!trd_mol<RT, CR, 1, false>((int)rank, (int)G, n, S.Fp + B.m_mat0[m], S.dtri + ao0, S.etri + ao0, S.tau + ao0,
                                   nullptr, &S.status[m]))
        atomicOr(&S.status[m], ST_TIMEOUT);
    if (cycles) trd_cycles(S, m, (int)rank, (int)G, t0, cycles);
}

// One molecule on the whole cooperative grid (every CTA resident, as its waits need); xpub: 4 n doubles and a count, zero
template <int RT, int CR>
__global__ void __launch_bounds__(TRD_THREADS, 1) k_trd_grid(Batch B, State S, int m, double* xpub, unsigned long long* cycles) {
    const long long t0 = clock64();
    if (!S.active[m]) return;  // uniform over the grid
    const int n = B.m_nao[m], ao0 = B.m_ao0[m];
    if (!trd_mol<RT, CR, 8, true>((int)blockIdx.x, (int)gridDim.x, n, S.Fp + B.m_mat0[m], S.dtri + ao0, S.etri + ao0,
                                  S.tau + ao0, xpub, &S.status[m]))
        atomicOr(&S.status[m], ST_TIMEOUT);
    if (cycles) trd_cycles(S, m, (int)blockIdx.x, (int)gridDim.x, t0, cycles);
}

// One molecule of `list` per team, gridDim.y teams of gridDim.x CTAs; xpub: `stride` doubles per entry of the
// list. A kernel of its own: with the molecule's number and addresses in registers instead of kernel
// parameters the one above took 16.4 ms instead of 16.0 at 2400 AOs.
template <int RT, int CR>
__global__ void __launch_bounds__(TRD_THREADS, 1)
    k_trd_teams(Batch B, State S, const int* list, double* xpub, long long stride, unsigned long long* cycles) {
    const long long t0 = clock64();
    const int m = list[blockIdx.y];
    if (!S.active[m]) {  // uniform over the team; the other teams' grid barrier counts these CTAs too
        cg::this_grid().sync();
        return;
    }
    const int n = B.m_nao[m], ao0 = B.m_ao0[m];
    if (!trd_mol<RT, CR, 8, true>((int)blockIdx.x, (int)gridDim.x, n, S.Fp + B.m_mat0[m], S.dtri + ao0, S.etri + ao0,
                                  S.tau + ao0, xpub + blockIdx.y * stride, &S.status[m]))
        atomicOr(&S.status[m], ST_TIMEOUT);
    if (cycles) trd_cycles(S, m, (int)blockIdx.x, (int)gridDim.x, t0, cycles);
}

}  // namespace axg
