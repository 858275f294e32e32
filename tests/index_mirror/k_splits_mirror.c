/* CPU replay of the indexing of the split FP64 products: k_zt_u, k_group_sums_dmma, k_hk (row tiles of MT x 16,
 * cell ranges, runs and gene ranges with their partial sums; k_dgen.cu) and k_pair_gram (three tile sizes, a list of
 * genes, persistent grids; k_dgemm.cu). Every global index of every copy and store, that every copied cell, gene and
 * row is met once, and that every output is written once. Prints "ok" or the first index out of place. With the
 * argument "odd" the cell ranges of k_zt_u start at odd cells, with "short" the partial sums' buffer lacks a value. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAX(a, b) ((a) > (b) ? (a) : (b))
#define MIN(a, b) ((a) < (b) ? (a) : (b))
#define UP(a, b) (((a) + (b)-1) / (b))
#define NEED(c, ...)                     \
  do {                                   \
    if (!(c)) {                          \
      fprintf(stderr, "%s: ", #c);       \
      fprintf(stderr, __VA_ARGS__);      \
      fprintf(stderr, "\n");             \
      exit(1);                           \
    }                                    \
  } while (0)
enum { BK = 16, S = BK + 4, BN = 128 };
static int odd, shrt;

static int row_tile(int rows) { return rows <= 16 ? 1 : rows <= 48 ? 3 : rows <= 80 ? 5 : 9; }

/* ---- k_zt_u: m columns x n genes over N cells in `splits` ranges ---- */
static void zt_u(int m, int n, int N, int MT, int splits) {
  const int ldN = UP(N, 32) * 32, rows = MT * 16, mt = UP(m, rows), nt = UP(n, BN);
  int per = UP(N, splits);
  per += odd ? !(per & 1) : per & 1;
  const long part = (long)splits * m * n - shrt;
  char* out = calloc((size_t)splits * m * n, 1);
  int* met = calloc(N, sizeof(int));
  for (int z = 0; z < splits; z++) {
    const int kb = MIN(N, z * per), ke = MIN(N, (z + 1) * per), nsl = ke > kb ? UP(ke - kb, BK) : 0;
    for (int s = 0; s < nsl; s++)
      for (int kc = 0; kc < BK; kc += 2) {
        const int k = kb + s * BK + kc, nb = k < ke ? (k + 1 < ke ? 2 : 1) : 0, src = MIN(k, ldN - 2);
        NEED(src % 2 == 0, "16-byte copy from cell %d", src);
        NEED(src + MAX(nb, 0) <= ldN, "cells %d..", src);
        if (nb) NEED(src == k, "cell %d copied for %d", src, k);
        for (int q = 0; q < nb; q++) met[k + q]++;
        for (int q = 0; q < 2; q++) NEED(MIN(k + q, N - 1) < N, "1/Omega");
      }
    for (int x = 0; x < mt; x++)
      for (int y = 0; y < nt; y++)
        for (int r = x * rows; r < MIN(m, (x + 1) * rows); r++)
          for (int j = y * BN; j < MIN(n, (y + 1) * BN); j++) {
            const long e = ((long)z * m + r) * n + j;
            NEED(e < part, "partial sum %ld of %ld", e, part);
            out[e]++;
          }
  }
  for (int i = 0; i < N; i++) NEED(met[i] == 1, "cell %d met %d times (N %d, %d ranges)", i, met[i], N, splits);
  for (long e = 0; e < (long)splits * m * n; e++) NEED(out[e] == 1, "sum %ld written %d times", e, out[e]);
  free(out);
  free(met);
}

/* ---- k_group_sums_dmma: ns runs of whole slices per group, and k_reduce_groups ---- */
static void group_sums(int m, int n, int n_grp, const int* start, int N, int MT, int ns) {
  const int ldN = UP(N, 32) * 32, rows = MT * 16;
  const long part = (long)n_grp * ns * n * m - shrt;
  int* met = calloc(N, sizeof(int));
  char* out = calloc((size_t)n_grp * ns * n * m, 1);
  for (int z = 0; z < n_grp * ns; z++) {
    const int grp = z / ns, c = z - grp * ns, g0 = start[grp], g1 = start[grp + 1];
    const int per = UP(UP(g1 - g0, BK), ns) * BK, kb = MIN(g1, g0 + c * per), ke = MIN(g1, kb + per);
    const int nsl = ke > kb ? UP(ke - kb, BK) : 0, last = MAX(ke - 1, 0);
    for (int s = 0; s < nsl; s++)
      for (int kc = 0; kc < BK; kc++) {
        const int k = kb + s * BK + kc;
        NEED(MIN(k, last) < ldN, "cell %d", k);
        if (k < ke) met[k]++;
      }
    for (int x = 0; x < UP(m, rows); x++)
      for (int r = x * rows; r < MIN(m, (x + 1) * rows); r++)
        for (int j = 0; j < n; j++) {
          const long e = ((long)z * n + j) * m + r;
          NEED(ns == 1 || e < part, "partial sum %ld", e);
          out[e]++;
        }
  }
  for (int i = 0; i < N; i++) NEED(met[i] == 1, "cell %d met %d times (%d runs)", i, met[i], ns);
  for (long e = 0; e < (long)n_grp * ns * n * m; e++) NEED(out[e] == 1, "sum %ld", e);
  free(met);
  free(out);
}

/* ---- k_hk: table rows ld, gene ranges of jper, 128-slot tiles ---- */
static void hk(int ld, int J, int n_grp, int tiles, int MT, int ns) {
  const int rows = MT * 16, jper = UP(UP(J, ns), BK) * BK;
  const long part = (long)ns * ld * tiles * 128 - shrt, tab = (long)J * n_grp * ld;
  int* met = calloc(J, sizeof(int));
  char* out = calloc((size_t)ns * ld * tiles * 128, 1);
  for (int sp = 0; sp < ns; sp++) {
    const int jb = sp * jper, je = MIN(J, jb + jper), nsl = je > jb ? UP(je - jb, BK) : 0;
    for (int s = 0; s < nsl; s++)
      for (int k = 0; k < BK; k++) {
        const int j = jb + s * BK + k;
        if (j < je) met[j]++;
        for (int x = 0; x < UP(ld, rows); x++)
          for (int r = 0; r < rows; r++) {
            const long e = ((long)MIN(j, J - 1) * n_grp + n_grp - 1) * ld + MIN(x * rows + r, ld - 1);
            NEED(e < tab, "table %ld", e);
          }
      }
    for (int z = 0; z < tiles; z++)
      for (int x = 0; x < UP(ld, rows); x++)
        for (int r = x * rows; r < MIN(ld, (x + 1) * rows); r++)
          for (int slot = 0; slot < 128; slot++) {
            const long e = (((long)sp * ld + r) * tiles + z) * 128 + slot;
            NEED(ns == 1 || e < part, "partial sum %ld", e);
            out[e]++;
          }
  }
  for (int j = 0; j < J; j++) NEED(met[j] == 1, "gene %d met %d times (%d ranges)", j, met[j], ns);
  for (long e = 0; e < (long)ns * ld * tiles * 128; e++) NEED(out[e] == 1, "sum %ld", e);
  free(met);
  free(out);
}

/* ---- k_pair_gram: TM x TN tiles, `live` genes of a list of J, `grid` blocks ---- */
static void pair_gram(int TM, int TN, int n_pairs, int J, int live, int N, int c0, int c1, int grid) {
  const int ldN = UP(N, 32) * 32, pad = UP(n_pairs, 128) * 128, tm = UP(n_pairs, TM), tn = UP(live, TN), group = 12;
  char* out = calloc((size_t)n_pairs * J, 1);
  for (int b = 0; b < grid; b++)
    for (int id = b; id < tm * tn; id += grid) {
      const int per = group * tn, grp = id / per, first = grp * group, gm = MIN(tm - first, group), r = id - grp * per;
      const int p0 = (first + r % gm) * TM, j0 = (r / gm) * TN;
      NEED(p0 < tm * TM && j0 < tn * TN, "tile %d", id);
      for (int s = 0; s < UP(c1 - c0, BK); s++) {
        for (int k = 0; k < BK; k++) {
          const long row = MIN(s * BK + k, c1 - c0 - 1), e = row * pad + p0 + TM - 2;
          NEED(e + 1 < (long)(c1 - c0) * pad && e % 2 == 0, "pair product %ld", e);
        }
        for (int part = 0; part < 8; part++) {
          const int i = c0 + s * BK + part * 2, nb = MAX(0, MIN(2, MIN(N, c1) - i)), src = MIN(i, ldN - 2);
          NEED(src % 2 == 0 && src + nb <= ldN && (!nb || src == i), "weights of cell %d", i);
        }
      }
      for (int p = p0; p < MIN(n_pairs, p0 + TM); p++)
        for (int k = j0; k < MIN(live, j0 + TN); k++) out[(size_t)p * J + (J - 1 - k)]++; /* a list in any order */
    }
  for (int p = 0; p < n_pairs; p++)
    for (int k = 0; k < J; k++) NEED(out[(size_t)p * J + (J - 1 - k)] == (k < live), "pair %d, gene %d", p, k);
  free(out);
}

int main(int argc, char** argv) {
  odd = argc > 1 && !strcmp(argv[1], "odd");
  shrt = argc > 1 && !strcmp(argv[1], "short");
  const int ms[] = {1, 16, 17, 48, 49, 80, 81, 144, 145, 200}, ns[] = {1, 127, 129}, Ns[] = {1, 15, 16, 17, 333, 1000};
  for (int a = 0; a < 10; a++)
    for (int b = 0; b < 3; b++)
      for (int c = 0; c < 6; c++) {
        const int sp[] = {1, 3, 8, 31};
        for (int d = 0; d < 4; d++) zt_u(ms[a], ns[b], Ns[c], ms[a] > 144 && d == 0 ? 3 : row_tile(ms[a]), sp[d]);
        int start[6] = {0, Ns[c] / 7, Ns[c] / 7, Ns[c] / 2, Ns[c] - Ns[c] / 9, Ns[c]};
        for (int d = 0; d < 4; d++) group_sums(ms[a], ns[b], 5, start, Ns[c], row_tile(ms[a]), sp[d]);
        for (int d = 1; d <= 16; d += 5) hk(ms[a], Ns[c], 3, 2, row_tile(ms[a]), d);
      }
  const int tiles[][2] = {{128, 128}, {64, 64}, {64, 16}}, np[] = {1, 63, 65, 129, 700, 2211}, Js[] = {1, 15, 17, 130};
  for (int t = 0; t < 3; t++)
    for (int a = 0; a < 6; a++)
      for (int b = 0; b < 4; b++)
        for (int c = 0; c < 6; c++) {
          const int grids[] = {1, 5, 100000};
          for (int d = 0; d < 3; d++) {
            pair_gram(tiles[t][0], tiles[t][1], np[a], Js[b], Js[b], Ns[c], 0, Ns[c], grids[d]);
            pair_gram(tiles[t][0], tiles[t][1], np[a], Js[b], UP(Js[b], 3), Ns[c], 0, Ns[c], grids[d]);
            if (Ns[c] > 128) pair_gram(tiles[t][0], tiles[t][1], np[a], Js[b], 1, Ns[c], 128, MIN(Ns[c], 256), grids[d]);
          }
        }
  printf("ok\n");
  return 0;
}
