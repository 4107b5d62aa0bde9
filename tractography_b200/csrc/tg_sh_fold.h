/* Generated by gen_sh_tables.py -- do not edit. */
/* Folded real symmetric SH coefficients (see gen_sh_tables.py): per band
 * limit, the terms dst += c[src] * r of the fold, in accumulation order, and
 * the block layout (m, part, parity, K, offset) of the folded vector. */
#ifndef TG_SH_FOLD_H
#define TG_SH_FOLD_H

#define TGSH_FN static inline
#define TGSH_TABLE static const

#define TGSH_NTERMS 175
/* per band limit 0, 2, .., 8: first term, term count, folded length */
TGSH_TABLE int TGSH_FOLD_RANGE[5][3] = {
    {0, 1, 1},   /* lmax 0 */
    {1, 7, 6},   /* lmax 2 */
    {8, 22, 15},   /* lmax 4 */
    {30, 50, 28},   /* lmax 6 */
    {80, 95, 45},   /* lmax 8 */
};
TGSH_TABLE unsigned char TGSH_FOLD_DST[TGSH_NTERMS] = {
    0, 1, 1, 0, 2, 3, 4, 5, 2, 2, 2, 1, 1, 0, 4, 4,
    3, 6, 6, 5, 8, 8, 7, 10, 10, 9, 11, 12, 13, 14, 3, 3,
    3, 3, 2, 2, 2, 1, 1, 0, 6, 6, 6, 5, 5, 4, 9, 9,
    9, 8, 8, 7, 12, 12, 12, 11, 11, 10, 15, 15, 15, 14, 14, 13,
    17, 17, 16, 19, 19, 18, 21, 21, 20, 23, 23, 22, 24, 25, 26, 27,
    4, 4, 4, 4, 4, 3, 3, 3, 3, 2, 2, 2, 1, 1, 0, 8,
    8, 8, 8, 7, 7, 7, 6, 6, 5, 12, 12, 12, 12, 11, 11, 11,
    10, 10, 9, 16, 16, 16, 16, 15, 15, 15, 14, 14, 13, 20, 20, 20,
    20, 19, 19, 19, 18, 18, 17, 23, 23, 23, 22, 22, 21, 26, 26, 26,
    25, 25, 24, 29, 29, 29, 28, 28, 27, 32, 32, 32, 31, 31, 30, 34,
    34, 33, 36, 36, 35, 38, 38, 37, 40, 40, 39, 41, 42, 43, 44,
};
TGSH_TABLE unsigned char TGSH_FOLD_SRC[TGSH_NTERMS] = {
    0, 0, 3, 3, 4, 2, 5, 1, 0, 3, 10, 3, 10, 10, 4, 11,
    11, 2, 9, 9, 5, 12, 12, 1, 8, 8, 13, 7, 14, 6, 0, 3,
    10, 21, 3, 10, 21, 10, 21, 21, 4, 11, 22, 11, 22, 22, 2, 9,
    20, 9, 20, 20, 5, 12, 23, 12, 23, 23, 1, 8, 19, 8, 19, 19,
    13, 24, 24, 7, 18, 18, 14, 25, 25, 6, 17, 17, 26, 16, 27, 15,
    0, 3, 10, 21, 36, 3, 10, 21, 36, 10, 21, 36, 21, 36, 36, 4,
    11, 22, 37, 11, 22, 37, 22, 37, 37, 2, 9, 20, 35, 9, 20, 35,
    20, 35, 35, 5, 12, 23, 38, 12, 23, 38, 23, 38, 38, 1, 8, 19,
    34, 8, 19, 34, 19, 34, 34, 13, 24, 39, 24, 39, 39, 7, 18, 33,
    18, 33, 33, 14, 25, 40, 25, 40, 40, 6, 17, 32, 17, 32, 32, 26,
    41, 41, 16, 31, 31, 27, 42, 42, 15, 30, 30, 43, 29, 44, 28,
};
TGSH_TABLE double TGSH_FOLD_R[TGSH_NTERMS] = {
    0x1.20dd750429b6dp-2, 0x1.20dd750429b6dp-2, -0x1.42f601a8c679bp-2, 0x1.e471027d29b68p-1,
    -0x1.17b14102b0694p+0, -0x1.17b14102b0694p+0, 0x1.17b14102b0694p-1, 0x1.17b14102b0694p-1,
    0x1.20dd750429b6dp-2, -0x1.42f601a8c679bp-2, 0x1.44f923a4aeedbp-2, 0x1.e471027d29b68p-1,
    -0x1.96376c8ddaa92p+1, 0x1.d9eb53fad46ffp+1, -0x1.17b14102b0694p+0, 0x1.00e9f3901edf5p+1,
    -0x1.2bbb9c2824049p+2, -0x1.17b14102b0694p+0, 0x1.00e9f3901edf5p+1, -0x1.2bbb9c2824049p+2,
    0x1.17b14102b0694p-1, -0x1.e471027d29b67p-2, 0x1.a7e2e22d847fap+1, 0x1.17b14102b0694p-1,
    -0x1.e471027d29b67p-2, 0x1.a7e2e22d847fap+1, -0x1.c5274a45d91d9p+0, -0x1.c5274a45d91d9p+0,
    0x1.406d8aa0d83a5p-1, 0x1.406d8aa0d83a5p-1, 0x1.20dd750429b6dp-2, -0x1.42f601a8c679bp-2,
    0x1.44f923a4aeedbp-2, -0x1.45796cbf7209dp-2, 0x1.e471027d29b68p-1, -0x1.96376c8ddaa92p+1,
    0x1.ab2f5ebb45acep+2, 0x1.d9eb53fad46ffp+1, -0x1.4063870c7441bp+4, 0x1.d5e74e9acca49p+3,
    -0x1.17b14102b0694p+0, 0x1.00e9f3901edf5p+1, -0x1.74e0af1cec1a8p+1, -0x1.2bbb9c2824049p+2,
    0x1.17a88355b113ep+4, -0x1.339fc3ab0f95dp+4, -0x1.17b14102b0694p+0, 0x1.00e9f3901edf5p+1,
    -0x1.74e0af1cec1a8p+1, -0x1.2bbb9c2824049p+2, 0x1.17a88355b113ep+4, -0x1.339fc3ab0f95dp+4,
    0x1.17b14102b0694p-1, -0x1.e471027d29b67p-2, 0x1.d7a8373d0a21dp-2, 0x1.a7e2e22d847fap+1,
    -0x1.094e9f1255b30p+3, 0x1.e66578f6f272ep+3, 0x1.17b14102b0694p-1, -0x1.e471027d29b67p-2,
    0x1.d7a8373d0a21dp-2, 0x1.a7e2e22d847fap+1, -0x1.094e9f1255b30p+3, 0x1.e66578f6f272ep+3,
    -0x1.c5274a45d91d9p+0, 0x1.61be296dc7996p+1, -0x1.4443a5f9f6f74p+3, -0x1.c5274a45d91d9p+0,
    0x1.61be296dc7996p+1, -0x1.4443a5f9f6f74p+3, 0x1.406d8aa0d83a5p-1, -0x1.025654a6adc03p-1,
    0x1.6336b4652ee84p+2, 0x1.406d8aa0d83a5p-1, -0x1.025654a6adc03p-1, 0x1.6336b4652ee84p+2,
    -0x1.2eed606fefa75p+1, -0x1.2eed606fefa75p+1, 0x1.5dca4e99e480ep-1, 0x1.5dca4e99e480ep-1,
    0x1.20dd750429b6dp-2, -0x1.42f601a8c679bp-2, 0x1.44f923a4aeedbp-2, -0x1.45796cbf7209dp-2,
    0x1.45ab7b94410ebp-2, 0x1.e471027d29b68p-1, -0x1.96376c8ddaa92p+1, 0x1.ab2f5ebb45acep+2,
    -0x1.6e60eb06c9308p+3, 0x1.d9eb53fad46ffp+1, -0x1.4063870c7441bp+4, 0x1.f7c5432954a2cp+5,
    0x1.d5e74e9acca49p+3, -0x1.b499e4df8d9e1p+6, 0x1.d3c97538aa04dp+5, -0x1.17b14102b0694p+0,
    0x1.00e9f3901edf5p+1, -0x1.74e0af1cec1a8p+1, 0x1.e881395e61963p+1, -0x1.2bbb9c2824049p+2,
    0x1.17a88355b113ep+4, -0x1.4fd8d770e3174p+5, -0x1.339fc3ab0f95dp+4, 0x1.b499e4df8d9e3p+6,
    -0x1.37dba37b1c035p+6, -0x1.17b14102b0694p+0, 0x1.00e9f3901edf5p+1, -0x1.74e0af1cec1a8p+1,
    0x1.e881395e61963p+1, -0x1.2bbb9c2824049p+2, 0x1.17a88355b113ep+4, -0x1.4fd8d770e3174p+5,
    -0x1.339fc3ab0f95dp+4, 0x1.b499e4df8d9e3p+6, -0x1.37dba37b1c035p+6, 0x1.17b14102b0694p-1,
    -0x1.e471027d29b67p-2, 0x1.d7a8373d0a21dp-2, -0x1.d31993dfe5dd3p-2, 0x1.a7e2e22d847fap+1,
    -0x1.094e9f1255b30p+3, 0x1.e1b2607ee50c1p+3, 0x1.e66578f6f272ep+3, -0x1.04eb499a11669p+6,
    0x1.04eb499a11669p+6, 0x1.17b14102b0694p-1, -0x1.e471027d29b67p-2, 0x1.d7a8373d0a21dp-2,
    -0x1.d31993dfe5dd3p-2, 0x1.a7e2e22d847fap+1, -0x1.094e9f1255b30p+3, 0x1.e1b2607ee50c1p+3,
    0x1.e66578f6f272ep+3, -0x1.04eb499a11669p+6, 0x1.04eb499a11669p+6, -0x1.c5274a45d91d9p+0,
    0x1.61be296dc7996p+1, -0x1.da579aa846684p+1, -0x1.4443a5f9f6f74p+3, 0x1.00ef73c5d0cddp+5,
    -0x1.81672da8b934bp+5, -0x1.c5274a45d91d9p+0, 0x1.61be296dc7996p+1, -0x1.da579aa846684p+1,
    -0x1.4443a5f9f6f74p+3, 0x1.00ef73c5d0cddp+5, -0x1.81672da8b934bp+5, 0x1.406d8aa0d83a5p-1,
    -0x1.025654a6adc03p-1, 0x1.e9e6057ed4466p-2, 0x1.6336b4652ee84p+2, -0x1.8e0ae4770c793p+3,
    0x1.f18d9d94cf977p+4, 0x1.406d8aa0d83a5p-1, -0x1.025654a6adc03p-1, 0x1.e9e6057ed4466p-2,
    0x1.6336b4652ee84p+2, -0x1.8e0ae4770c793p+3, 0x1.f18d9d94cf977p+4, -0x1.2eed606fefa75p+1,
    0x1.b996abd80466ep+1, -0x1.13fe2b6702c05p+4, -0x1.2eed606fefa75p+1, 0x1.b996abd80466ep+1,
    -0x1.13fe2b6702c05p+4, 0x1.5dca4e99e480ep-1, -0x1.108deb99a141bp-1, 0x1.ff0a19c00e5b2p+2,
    0x1.5dca4e99e480ep-1, -0x1.108deb99a141bp-1, 0x1.ff0a19c00e5b2p+2, -0x1.7535e00d444d1p+1,
    -0x1.7535e00d444d1p+1, 0x1.7535e00d444d1p-1, 0x1.7535e00d444d1p-1,
};

/* Block layout for band limit 8; a smaller band limit L keeps the blocks
 * with m <= L, each with K = (L - m - parity) / 2 + 1, packed in order. */
#define TGSH_NBLOCKS 17
TGSH_TABLE int TGSH_BLOCKS[TGSH_NBLOCKS][2] = {   /* m, part (0 cos, 1 sin) */
    {0, 0},
    {1, 0},
    {1, 1},
    {2, 0},
    {2, 1},
    {3, 0},
    {3, 1},
    {4, 0},
    {4, 1},
    {5, 0},
    {5, 1},
    {6, 0},
    {6, 1},
    {7, 0},
    {7, 1},
    {8, 0},
    {8, 1},
};

/* Fold the coefficients c (zero-padded to the full band of lmax) into a:
 * each a[d] is the double sum of its terms in table order, rounded once. */
TGSH_FN void tgsh_fold(int lmax, const float* c, float* a)
{
    const int* range = TGSH_FOLD_RANGE[lmax / 2];
    double acc[48];
    for (int i = 0; i < range[2]; ++i) acc[i] = 0.0;
    for (int t = range[0]; t < range[0] + range[1]; ++t) {
        const double prod = (double)c[TGSH_FOLD_SRC[t]] * TGSH_FOLD_R[t];
        acc[TGSH_FOLD_DST[t]] = acc[TGSH_FOLD_DST[t]] + prod;
    }
    for (int i = 0; i < range[2]; ++i) a[i] = (float)acc[i];
}

#endif
