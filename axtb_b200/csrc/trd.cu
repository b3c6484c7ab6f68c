// The tridiagonal reduction's kernels, one per size class (a translation unit of their own: ~50
// instances whose compilation runs beside the engine's).
#include "trd.cuh"

namespace axg {

// cluster path: rt = ceil(n / 32) exactly; rt x cr values of the matrix per thread leave the other
// ~90 of 255 registers to the pass. For clusters of G CTAs whose warps have few columns (clusters that
// grew) a class with all of them in registers and nothing unrolled for columns that are not there.
const TrdClass* trd_class(int n, int G) {
#define TRD_C(RT, CR) {RT, CR, (const void*)k_trd<RT, CR>, nullptr}
    static const TrdClass c[] = {TRD_C(1, 4),  TRD_C(2, 8),  TRD_C(3, 12), TRD_C(4, 16), TRD_C(5, 13), TRD_C(6, 12), TRD_C(7, 10), TRD_C(8, 9),  TRD_C(9, 8),
                                 TRD_C(10, 7), TRD_C(11, 7), TRD_C(12, 6), TRD_C(13, 6), TRD_C(14, 5), TRD_C(15, 5),
                                 TRD_C(16, 5), TRD_C(17, 4), TRD_C(18, 4), TRD_C(19, 4), TRD_C(20, 4), TRD_C(21, 3),
                                 TRD_C(22, 3), TRD_C(23, 3), TRD_C(24, 3)};
    static const TrdClass f[] = {TRD_C(1, 4),  TRD_C(2, 4),  TRD_C(3, 4),  TRD_C(4, 4),  TRD_C(5, 4),  TRD_C(6, 4),  TRD_C(7, 4),  TRD_C(8, 4),  TRD_C(9, 4),
                                 TRD_C(10, 4), TRD_C(11, 4), TRD_C(12, 4), TRD_C(13, 4), TRD_C(14, 4), TRD_C(15, 4),
                                 TRD_C(16, 4), TRD_C(17, 5), TRD_C(18, 5), TRD_C(19, 5)};
#undef TRD_C
    const int rt = (n + 31) / 32;
    if (rt < 1 || rt > 24) return nullptr;
    return G > 0 && rt <= 19 && trd_slots(n, G, 8) <= f[rt - 1].cr ? f + (rt - 1) : c + (rt - 1);
}
// whole grid: n <= 256 rt
const TrdClass* trd_grid_class(int n) {
#define TRD_C(RT, CR) {RT, CR, (const void*)k_trd_grid<RT, CR>, nullptr}
#define TRD_T(RT, CR) {RT, CR, (const void*)k_trd_grid<RT, CR>, (const void*)k_trd_teams<RT, CR>}
    static const TrdClass c[] = {TRD_T(4, 8), TRD_T(5, 9), TRD_T(6, 11), TRD_T(7, 11), TRD_C(8, 9), TRD_C(10, 9)};
#undef TRD_T
#undef TRD_C
    for (const TrdClass& x : c)
        if (n <= 256 * x.rt) return &x;
    return nullptr;
}

}  // namespace axg
