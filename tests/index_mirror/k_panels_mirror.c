/* CPU replay of the indexing of the panel kernels of k_inv.cu (k_potrf_panel, k_potrf_rows, k_tri_diag,
 * k_trtri_panel, k_lauum_panel and the ring of k_irls_tail): every shared- and global-memory index of every thread,
 * which chunk or block a buffer holds when it is read, whether a copied column is finished by then, and how
 * often each output is written. The block sizes come from the source (-D). Usage: k_panels_mirror kernel from to;
 * prints "ok kernel from..to" or the first index out of place. */
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#define MAX(a, b) ((a) > (b) ? (a) : (b))
#define MIN(a, b) ((a) < (b) ? (a) : (b))
static int P;
static const char* at;
#define NEED(c, ...)                                      \
  do {                                                    \
    if (!(c)) {                                           \
      fprintf(stderr, "%s P=%d: %s: ", at, P, #c);        \
      fprintf(stderr, __VA_ARGS__);                       \
      fprintf(stderr, "\n");                              \
      exit(1);                                            \
    }                                                     \
  } while (0)

/* one copy of n doubles from A[src ..] (none: a zero fill) to shared dst .. within [lo, hi) */
static void copy(long src, long dst, int n, int filled, long lo, long hi) {
  NEED(dst >= lo && dst + n <= hi, "copy to %ld in [%ld, %ld)", dst, lo, hi);
  if (n == 2) NEED(dst % 2 == 0 && src % 2 == 0, "16-byte copy from %ld to %ld", src, dst);
  NEED(src >= 0 && src + (filled ? n : 0) <= (long)P * P, "copy from %ld", src);
}

/* ---- k_potrf_panel ---- */
static int panel_smem(int ns) {
  const int rp = MAX(IB, (P + 15) / 16 * 16);
  return 8 * (IB * (rp + 2) + ns * CW * (rp + 4) + IB);
}
static int buffers(int extra) { return 2 * (panel_smem(3) + extra + 1536) <= 228 * 1024 ? 3 : 2; }

static int p0, rpad, SA, cw, nbuf, lch, lbuf, holds[4], finished, warps;
static long La, La_end;
static void column(long dst, int col, int ok, long lo, long hi) {
  const int pairs = P % 2 == 0, rows = P - p0;
  const long src = p0 + (long)(ok ? col : 0) * P;
  for (int lane = 0; lane < 32; lane++)
    for (int r = (pairs ? 2 : 1) * lane; r < rpad; r += pairs ? 64 : 32) {
      const int f = ok && r < rows;
      copy(f ? src + r : src, dst + r, pairs ? 2 : 1, f, lo, hi);
      if (f && pairs) NEED(r + 1 < rows, "row %d of a pair past the matrix", r + 1);
    }
}
static void panel(int c0, long space) {
  p0 = c0;
  rpad = (P - c0 + 15) / 16 * 16;
  SA = MAX(IB, rpad) + 4;
  cw = IB;
  while (cw > CW && 2 * cw * SA > space) cw >>= 1;
  nbuf = 3 * cw * SA <= space ? 3 : 2;
  lch = lbuf = 0;
  NEED((long)nbuf * cw * SA <= space, "%d chunks of %d columns", nbuf, cw);
  NEED(SA % 2 == 0 && IB % cw == 0 && cw % 4 == 0, "chunk shape");
  for (int k = 0; k < 4; k++) holds[k] = -1;
}
static void stage(int reading) {
  if (lch < p0 / cw) {
    NEED(lbuf != reading, "buffer %d refilled while it is read", lbuf);
    for (int q = 0; q < cw; q++) {
      NEED(lch * cw + q < finished, "column %d copied before it is finished (%d)", lch * cw + q, finished);
      column(La + (long)(lbuf * cw + q) * SA, lch * cw + q, 1, La, La_end);
    }
    holds[lbuf] = lch++;
    lbuf = lbuf + 1 == nbuf ? 0 : lbuf + 1;
  }
}
static void potrf(int T) {
  const int ns = buffers(0), rp = MAX(IB, (P + 15) / 16 * 16), SP = rp + 2;
  const long space = (long)ns * CW * (rp + 4);
  NEED(panel_smem(ns) <= 220 * 1024, "%d bytes", panel_smem(ns));
  warps = T / 32;
  La = (long)IB * SP;
  La_end = La + space;
  finished = 0;
  char* out = calloc((size_t)P * P, 1);
  panel(0, space);
  for (int c0 = 0; c0 < P; c0 += IB) {
    const int rows = P - c0, ncol = MIN(IB, rows), nch = c0 / cw;
    NEED(p0 == c0, "panel %d", p0);
    for (int k = lch; k < nbuf - 1; k++) stage(-1);
    for (int cc = 0; cc < IB; cc++) column((long)cc * SP, c0 + cc, cc < ncol, 0, La);
    for (int ch = 0, buf = 0; ch < nch; ch++) {
      NEED(holds[buf] == ch, "buffer %d holds chunk %d at step %d", buf, holds[buf], ch);
      stage(buf);
      buf = buf + 1 == nbuf ? 0 : buf + 1;
    }
    NEED(nch == 0 || nch * cw == c0, "chunks cover the finished columns");
    int* hit = calloc(rpad, sizeof(int)); /* rows of the panel's update */
    for (int w = 0; w < warps; w++)
      for (int x = 0; x < 2; x++) {
        const int mt = w + warps * x;
        if (mt * 16 >= rpad) continue;
        for (int g = 0; g < 16; g++) {
          NEED(mt * 16 + g < SA && mt * 16 + g < SP, "row %d", mt * 16 + g);
          hit[mt * 16 + g]++;
        }
      }
    for (int r = 0; r < rows && nch > 0; r++) NEED(hit[r] == 1, "row %d updated %d times", r, hit[r]);
    free(hit);
    if (c0 + IB < P) {
      panel(c0 + IB, space);
      while (lch < nbuf - 1 && (lch + 1) * cw <= c0) stage(-1);
    }
    for (int cc = 0; cc < ncol; cc++)
      for (int r = cc; r < rows; r++) {
        NEED((long)cc * SP + r < La, "store from row %d", r);
        out[(size_t)(c0 + r) + (size_t)(c0 + cc) * P]++;
      }
    finished = c0 + IB;
  }
  for (int c = 0; c < P; c++)
    for (int r = c; r < P; r++) NEED(out[r + (size_t)c * P] == 1, "entry (%d, %d) written %d times", r, c, out[r + (size_t)c * P]);
  free(out);
  /* the ring of k_irls_tail in the panel's space: 16 columns, rows to P (to the next even one in pairs) */
  const int RS = rp + 2;
  for (int k = 0; k < P; k++) {
    const int from = P % 2 == 0 ? (k + 1) & ~1 : k + 1;
    for (int r = from; r < P; r += P % 2 == 0 ? 2 : 1)
      copy((long)k * P + r, (long)(k % 16) * RS + r, P % 2 == 0 ? 2 : 1, 1, 0, (long)IB * SP);
  }
}

/* ---- k_potrf_rows ---- */
static void potrf_rows(void) {
  const int RSA = RB + 4, RSB = IB + 4, even = P % 2 == 0;
  const long oLa = (long)RB * IS, oLb = oLa + 2L * RC * RSA, oDg = oLb + 2L * RC * RSB, oRd = oDg + IB * (IB + 2);
  NEED(8 * (oRd + IB) <= 220 * 1024, "%ld bytes", 8 * (oRd + IB));
  char* out = calloc((size_t)P * P, 1);
  for (int c0 = 0; c0 < P; c0 += IB) {
    const int ncol = MIN(IB, P - c0);
    for (int r0 = c0; r0 < P; r0 += RB) {
      const int rows = MIN(RB, P - r0);
      NEED(c0 % RC == 0, "chunks");
      for (int ch = 0; ch < c0 / RC; ch++)
        for (int q = 0; q < RC; q++)
          for (int r = 0; r < RB + IB; r += even ? 2 : 1) {
            const int a = r < RB, row = a ? r0 + r : c0 + r - RB, n = even ? 2 : 1;
            const long src = (long)(ch * RC + q) * P + MIN(row, P - n);
            const long dst = a ? oLa + (long)(ch & 1) * RC * RSA + q * RSA + r : oLb + (long)(ch & 1) * RC * RSB + q * RSB + r - RB;
            copy(src, dst, n, 1, a ? oLa : oLb, a ? oLb : oDg);
            if (row < P) NEED(row + n <= P, "row %d", row);
            NEED(ch * RC + q < c0, "column %d not finished", ch * RC + q);
          }
      for (int r = 0; r < rows; r++)
        for (int cc = 0; cc < ncol; cc++)
          if (r0 > c0 || r >= cc) {
            NEED((long)r * IS + cc < oLa, "row %d", r);
            out[(size_t)(r0 + r) + (size_t)(c0 + cc) * P]++;
          }
    }
  }
  for (int c = 0; c < P; c++)
    for (int r = c; r < P; r++) NEED(out[r + (size_t)c * P] == 1, "entry (%d, %d)", r, c);
  free(out);
}

/* ---- the inverse: the stream of 32 x 32 blocks through NB buffers ---- */
static int sr[8], sc[8], s_buf; /* the block that each buffer holds */
static void block(int r, int c, long lo) { /* stage_block */
  for (int t = 0; t < 256; t++) {
    if (P % 2 == 0)
      for (int k = 0; k < 2; k++) {
        const int e = t + 256 * k, q = e >> 4, m = 2 * (e & 15), ok = r + m < P && c + q < P;
        copy(ok ? (long)(r + m) + (long)(c + q) * P : 0, lo + q * IS + m, 2, ok, lo, lo + IB * IS);
        if (ok) NEED(r + m + 1 < P, "row %d", r + m + 1);
      }
    else
      for (int k = 0; k < 4; k++) {
        const int e = t + 256 * k, q = e >> 5, m = e & 31, ok = r + m < P && c + q < P;
        copy(ok ? (long)(r + m) + (long)(c + q) * P : 0, lo + q * IS + m, 1, ok, lo, lo + IB * IS);
      }
  }
}
static void inverse(int lauum) {
  const int nb = (P + IB - 1) / IB, SY = nb * IB + 4;
  const long oR = (long)IB * SY, oS = lauum ? oR : oR + IB * IS, end = oS + (long)NB * IB * IS;
  NEED(8 * end <= 8L * (IB * (nb * IB + 4) + IB * IS + NB * IB * IS) && 8 * end <= 220 * 1024, "%ld bytes", 8 * end);
  char* out = calloc((size_t)P * P, 1);
  for (int b = 0; b < (lauum ? nb : nb - 1); b++) {
    int li = b + 1, lc = b, la = b, lk = b;
    s_buf = 0;
    for (int k = 0; k < 8; k++) sr[k] = sc[k] = -1;
#define LOAD()                                                       \
  do {                                                               \
    if (lauum ? la < nb : li < nb) {                                 \
      sr[s_buf] = lauum ? lk : li;                                   \
      sc[s_buf] = lauum ? la : lc;                                   \
      block(sr[s_buf] * IB, sc[s_buf] * IB, oS + (long)s_buf * IB * IS); \
      if (lauum) {                                                   \
        if (++lk == nb) lk = ++la;                                   \
      } else if (++lc > li) {                                        \
        li++;                                                        \
        lc = b;                                                      \
      }                                                              \
      s_buf = s_buf + 1 == NB ? 0 : s_buf + 1;                       \
    }                                                                \
  } while (0)
    for (int k = 0; k < NB - 1; k++) LOAD();
    int buf = 0;
    if (lauum) {
      for (int n = 0; n < IB; n++)
        for (int k = 0; k < (nb - b) * IB; k++) NEED((long)n * SY + k < oR, "panel row %d", k);
      for (int a = b; a < nb; a++)
        for (int kc = a; kc < nb; kc++) {
          NEED(s_buf != buf || la >= nb, "buffer refilled");
          LOAD();
          NEED(sr[buf] == kc && sc[buf] == a, "buffer holds (%d, %d), not (%d, %d)", sr[buf], sc[buf], kc, a);
          NEED((long)31 * SY + (kc - b) * IB + 31 < oR, "panel");
          buf = buf + 1 == NB ? 0 : buf + 1;
          if (kc == nb - 1)
            for (int m = 0; m < IB; m++)
              for (int n = 0; n < IB; n++) {
                const int row = a * IB + m, col = b * IB + n;
                if (row < P && col < P) {
                  out[(size_t)row + (size_t)col * P] |= 1;
                  out[(size_t)col + (size_t)row * P] |= 1;
                }
              }
        }
    } else {
      for (int i = b + 1; i < nb; i++)
        for (int ch = b; ch <= i; ch++) {
          LOAD();
          NEED(sr[buf] == i && sc[buf] == ch, "buffer holds (%d, %d), not (%d, %d)", sr[buf], sc[buf], i, ch);
          NEED((long)31 * SY + (i - b) * IB + 31 < oR, "solution");
          buf = buf + 1 == NB ? 0 : buf + 1;
        }
      for (int n = 0; n < MIN(IB, P - b * IB); n++)
        for (int r = IB; r < P - b * IB; r++) {
          NEED((long)n * SY + r < oR, "row %d", r);
          out[(size_t)(b * IB + r) + (size_t)(b * IB + n) * P]++;
        }
    }
  }
  for (int c = 0; c < P; c++)
    for (int r = 0; r < P; r++) {
      const int want = lauum || r / IB > c / IB;
      NEED(out[r + (size_t)c * P] == want, "entry (%d, %d) written %d times", r, c, out[r + (size_t)c * P]);
    }
  free(out);
}

int main(int argc, char** argv) {
  if (argc != 4) return 2;
  at = argv[1];
  const int from = atoi(argv[2]), to = atoi(argv[3]);
  for (P = from; P <= to; P++) {
    if (!strcmp(at, "potrf")) potrf(P <= kPotrfHalfP ? 128 : 256);
    else if (!strcmp(at, "rows")) potrf_rows();
    else if (!strcmp(at, "trtri")) inverse(0);
    else if (!strcmp(at, "lauum")) inverse(1);
    else return 2;
  }
  printf("ok %s %d..%d\n", at, from, to);
  return 0;
}
