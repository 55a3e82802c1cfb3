// Test helper: the layout rules of the resident integrator (kura_resident.cuh) on the host, over all
// shapes.  Prints the first violations and exits 1; no GPU is used.
#include <cstdio>
#include <cstring>
#include "kura_resident.cuh"

using namespace kura;

static int bad = 0;
static void fail(const char* what, const ResSplit& s, int a, int b) {
  if (++bad <= 5) printf("%s: B %d k %d blocks %d rows %d den %d: %d %d\n", what, s.B, s.k, s.vblocks, s.vrows, s.den, a, b);
}
// the grid of the persistent kernel on `sms` multiprocessors
static ResSplit split(int n, int B, int k, int den, int sms) {
  const int least = den ? 16 : 64;
  int G = (n + least - 1) / least;
  if (G > sms) G = sms;
  const int rows = (n + G - 1) / G;
  G = (n + rows - 1) / rows;
  return {B, k, rows, rows, G, G, den, (n + 31) / 32 * 32};
}
template <class F>
static void all_shapes(F f) {
  for (int sms : {152, 148, 132, 20})
    for (int n = 1; n < 12000; n += n < 700 ? 1 : 37)
      for (int k = 0; k <= 8; ++k)
        for (int B = 1; B <= 8; ++B) {
          f(split(n, B, k, 0, sms));
          if (B == 1 && k == 0) f(split(n, 1, 0, RES_F32, sms));
        }
}

// the sums of an exchange that a slow CTA still reads are not written by the next exchange, whose
// number of sums may be another, and every half lies in the buffer (2 * blocks * B * PW_MAX floats)
static void part() {
  all_shapes([](const ResSplit& s) {
    const int per[] = {1, 2, s.k ? 2 * s.k : 1, RES_RED};
    for (int first : per)
      for (int next : per)
        for (int par = 0; par < 2; ++par) {
          const int nv = first * s.B, nw = next * s.B;
          const size_t a0 = res_part(s, par, 0, nv), a1 = res_part(s, par, s.vblocks - 1, nv) + nv;
          const size_t b0 = res_part(s, par ^ 1, 0, nw), b1 = res_part(s, par ^ 1, s.vblocks - 1, nw) + nw;
          if (a0 < b1 && b0 < a1) fail("halves overlap", s, nv, nw);
          if (a1 > 2 * (size_t)s.vblocks * s.B * PW_MAX) fail("past the buffer", s, nv, (int)a1);
        }
  });
}

// the slices of ordered sums fit their buffer in every kind of pass
static void slices() {
  all_shapes([](const ResSplit& s) {
    int off[18];
    for (int mode : {RES_ONE, RES_CLUSTER, RES_GRIDX}) {
      if (mode != RES_GRIDX && (s.den || s.vrows * s.vblocks * s.B > 12288)) continue;
      if (mode == RES_ONE && s.vblocks > 4) continue;
      ResSplit t = s;
      t.ctas = mode == RES_ONE ? 1 : mode == RES_CLUSTER ? (s.vblocks < 16 ? s.vblocks : 16) : s.vblocks;
      t.rows = (s.vblocks + t.ctas - 1) / t.ctas * s.vrows;
      res_layout(t, 1, mode, 512, off);
      const int room = (off[7] - off[6]) / 4;
      for (int kind : {0, 2, 8, 9})
        for (int flags = 0; flags < 4; ++flags) {
          const ResSums q = res_sums(kind, s.k, s.den != 0, flags & 1, flags & 2);
          const int S = res_slices(s.vblocks, q.npw), need = S > 1 ? S * s.B * q.nv : 0;
          if (need > room) fail("slices", s, need, room);
        }
    }
  });
}

int main(int argc, char** argv) {
  const char* what = argc > 1 ? argv[1] : "";
  if (!strcmp(what, "part")) part();
  else if (!strcmp(what, "slices")) slices();
  else return 2;
  printf("%d violations\n", bad);
  return bad != 0;
}
