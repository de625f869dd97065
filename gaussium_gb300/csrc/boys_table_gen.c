/*
 * Writes the Boys-function grid used by the ERI kernels as a C header of hexadecimal
 * floating-point literals (exact), computed in long double:
 *
 *   row k (T_k = k / BOYS_INV_H, k = 0..BOYS_ROWS-1):
 *     col m = F_m(T_k) for m = 0..BOYS_NCOL-2,   col BOYS_NCOL-1 = exp(-T_k)
 *
 * F_top(T) comes from the series F_m(T) = exp(-T) sum_i (2T)^i / ((2m+1)(2m+3)...(2m+2i+1)),
 * whose terms are all positive, and the lower orders from the downward recursion
 * F_{m-1} = (2T F_m + exp(-T)) / (2m-1), which is stable.  The kernels evaluate
 * F_m(T) by a Taylor expansion about the nearest grid point and the downward recursion
 * (Helgaker, Jorgensen & Olsen, Molecular Electronic-Structure Theory, sec. 9.8.2).
 * The grid reaches T = 80, beyond which exp(-T) < 2e-35 changes no F_m (m <= 16) in double
 * precision, so the kernels' large-T branch needs no exponential.
 *
 * It also writes Taylor rows per order M = 0..BOYS_TAYLOR_MMAX on a grid of half the step
 * up to one past the order's asymptotic threshold (GS_BOYS_ROW64_<M>: row k, T_k =
 * k / BOYS_INV_H64, is {{F_{M+j}(T_k) / j!, j = 0..3},
 * {exp(-T_k) / j!, j = 0..3}, {F_{M+j}(T_k) / j!, j = 4..6 and a zero, float},
 * {exp(-T_k) / j!, j = 4..6 and a zero, float}}): with the factorials folded in, an expansion
 * about T_k is a Horner chain of FMAs in T_k - T.  The terms from the fourth on are at most
 * (1/64)^4 / 4! = 2^-28.6 of the value, so their rounding to float is 2^-52.6 of it.
 *
 * For FP32 quartets (T below BOYS_TMAX32, their largest asymptotic threshold) it writes
 * GS_BOYS_F32_<M>: row k = twelve floats {hi, lo of F_M(T_k); hi, lo of F_{M+1}(T_k);
 * F_{M+j}(T_k) / j!, j = 2..4; 0; hi, lo of exp(-T_k); 0, 0}, hi + lo being the value to twice a
 * float's precision.
 *
 * usage: boys_table_gen OUT.h
 */
#include <math.h>
#include <stdio.h>

#define BOYS_INV_H 16
#define BOYS_TMAX 80
#define BOYS_ROWS (BOYS_TMAX * BOYS_INV_H + 1)
#define BOYS_NCOL 18 /* F_0..F_16 and exp(-T) */
#define BOYS_INV_H64 32
#define BOYS_ROWS64 (BOYS_TMAX * BOYS_INV_H64 + 1)
#define BOYS_TMAX32 50
#define BOYS_TAYLOR_MMAX 10 /* F_{M+6} is the highest order tabulated */

/* asymptotic thresholds of orders 0..BOYS_TAYLOR_MMAX (kBoysAsym64 in eri_common.cuh) */
static const int asym64[BOYS_TAYLOR_MMAX + 1] = {36, 40, 43, 46, 49, 52, 54, 57, 59, 61, 64};

static void pair32(FILE *f, long double x)
{
    const float hi = (float)x;
    fprintf(f, "%af,%af,", hi, (float)(x - hi));
}

/* F[0..BOYS_NCOL-2] = F_m(T) and F[BOYS_NCOL-1] = exp(-T). */
static void boys_all(long double T, long double *F)
{
    const int top = BOYS_NCOL - 2;
    long double e = expl(-T);
    long double term = 1.0L / (2 * top + 1), sum = term;
    for (int i = 1; i < 100000; ++i) {
        term *= 2.0L * T / (2 * top + 2 * i + 1);
        sum += term;
        if (term < sum * 1e-24L) break;
    }
    F[top] = e * sum;
    for (int m = top; m >= 1; --m) F[m - 1] = (2.0L * T * F[m] + e) / (2 * m - 1);
    F[BOYS_NCOL - 1] = e;
}

int main(int argc, char **argv)
{
    if (argc != 2) return 2;
    FILE *f = fopen(argv[1], "w");
    if (!f) return 1;
    fprintf(f, "// generated by boys_table_gen.c -- Boys function grid\n#pragma once\n");
    fprintf(f, "#define BOYS_INV_H %d\n#define BOYS_TMAX %d\n#define BOYS_ROWS %d\n#define BOYS_NCOL %d\n",
            BOYS_INV_H, BOYS_TMAX, BOYS_ROWS, BOYS_NCOL);
    static long double F[BOYS_ROWS][BOYS_NCOL], H[BOYS_ROWS64][BOYS_NCOL];
    for (int k = 0; k < BOYS_ROWS; ++k) boys_all((long double)k / BOYS_INV_H, F[k]);
    for (int k = 0; k < BOYS_ROWS64; ++k) boys_all((long double)k / BOYS_INV_H64, H[k]);
    fprintf(f, "#define BOYS_TAYLOR_MMAX %d\n", BOYS_TAYLOR_MMAX);
    fprintf(f, "#define GS_BOYS_TABLE_VALUES \\\n");
    for (int k = 0; k < BOYS_ROWS; ++k) {
        for (int m = 0; m < BOYS_NCOL; ++m) fprintf(f, "%a,", (double)F[k][m]);
        fprintf(f, " \\\n");
    }
    fprintf(f, "\n");
    long double fact[7] = {1, 1, 2, 6, 24, 120, 720};
    fprintf(f, "#define BOYS_INV_H64 %d\n", BOYS_INV_H64);
    for (int M = 0; M <= BOYS_TAYLOR_MMAX; ++M) {
        fprintf(f, "#define GS_BOYS_ROW64_%d \\\n", M);
        for (int k = 0; k <= (asym64[M] + 1) * BOYS_INV_H64; ++k) {
            const long double *r = H[k], e = r[BOYS_NCOL - 1];
            fprintf(f, "{{%a,%a,%a,%a},", (double)r[M], (double)r[M + 1],
                    (double)(r[M + 2] / fact[2]), (double)(r[M + 3] / fact[3]));
            fprintf(f, "{%a,%a,%a,%a},", (double)e, (double)e, (double)(e / fact[2]),
                    (double)(e / fact[3]));
            fprintf(f, "{%af,%af,%af,0.0f},", (float)(r[M + 4] / fact[4]),
                    (float)(r[M + 5] / fact[5]), (float)(r[M + 6] / fact[6]));
            fprintf(f, "{%af,%af,%af,0.0f}}, \\\n", (float)(e / fact[4]), (float)(e / fact[5]),
                    (float)(e / fact[6]));
        }
        fprintf(f, "\n");
    }
    fprintf(f, "\n#define BOYS_TMAX32 %d\n#define BOYS_ROWS32 %d\n", BOYS_TMAX32,
            BOYS_TMAX32 * BOYS_INV_H + 1);
    for (int M = 0; M <= BOYS_TAYLOR_MMAX; ++M) {
        fprintf(f, "#define GS_BOYS_F32_%d \\\n", M);
        for (int k = 0; k <= BOYS_TMAX32 * BOYS_INV_H; ++k) {
            pair32(f, F[k][M]);
            pair32(f, F[k][M + 1]);
            for (int j = 2; j <= 4; ++j) fprintf(f, "%af,", (float)(F[k][M + j] / fact[j]));
            fprintf(f, "0.0f,");
            pair32(f, F[k][BOYS_NCOL - 1]);
            fprintf(f, "0.0f,0.0f, \\\n");
        }
        fprintf(f, "\n");
    }
    fclose(f);
    return 0;
}
