/* The 6x6 linear solve of the tangent kernels. */
#ifndef ATB_SOLVE6_CUH
#define ATB_SOLVE6_CUH

namespace atb {

/* w = J^-1 g for M = (J | g): Gaussian elimination with partial pivoting held
 * in registers.  Row swaps are selects and every loop has constant bounds, so
 * that every index is known when the array is split into registers (with
 * triangular loop bounds it stayed in local memory: 230 stores and 170 loads a
 * solve, a fifth of the tangent kernel's time). */
__device__ __forceinline__ void solve6(double (&M)[6][7], double w[6]) {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        /* pivot: the largest |M[i][c]|, i >= c */
        double best = fabs(M[c][c]);
        int piv = c;
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            if (i > c) {
                const double a = fabs(M[i][c]);
                if (a > best) { best = a; piv = i; }
            }
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            if (i > c) {
                const bool sw = (piv == i);
#pragma unroll
                for (int j = 0; j < 7; ++j) {
                    if (j >= c) {
                        const double t = M[c][j];
                        M[c][j] = sw ? M[i][j] : t;
                        M[i][j] = sw ? t : M[i][j];
                    }
                }
            }
        }
        const double inv = 1.0 / M[c][c];
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            if (i > c) {
                const double f = M[i][c] * inv;
#pragma unroll
                for (int j = 0; j < 7; ++j)
                    if (j > c) M[i][j] -= f * M[c][j];
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        const int i = 5 - k;
        double s = M[i][6];
#pragma unroll
        for (int j = 0; j < 6; ++j)
            if (j > i) s -= M[i][j] * w[j];
        w[i] = s / M[i][i];
    }
}

}  // namespace atb

#endif  // ATB_SOLVE6_CUH
