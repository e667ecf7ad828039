/* Host driver of the fixed-point row's functions as the row assembly uses them
   (fx.cuh) for tests/test_fx_rows_host.py: reads from argv[1] a row of nc
   contributions of one table (header: nc, nen, nblk, den; per contribution the
   row slot a, 16 block targets and D 15x15; the 5x16 table; three pressure
   vectors of the corners 0..2 per contribution) and sums them in the row's unit
   and in double with every element in its own (fx_wide); writes the row's
   exponents (9), whether the rule keeps the row in integers, and both rows,
   the first as integers in two words. */
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <vector>

#include "../biofem-ia_gb300/csrc/fx.cuh"

using namespace biofem;

int main(int argc, char **argv)
{
  if (argc != 3) return 2;
  FILE *f = std::fopen(argv[1], "rb");
  if (!f) return 3;
  int h[4];
  if (std::fread(h, sizeof(int), 4, f) != 4) return 4;
  const int nc = h[0], nen = h[1], nblk = h[2], den = h[3];
  std::vector<int> a(nc), tgt((size_t)nc * 16);
  std::vector<double> D((size_t)nc * 225), N(80), P((size_t)nc * 9);
  if (std::fread(a.data(), sizeof(int), nc, f) != (size_t)nc || std::fread(tgt.data(), sizeof(int), tgt.size(), f) != tgt.size() ||
      std::fread(D.data(), sizeof(double), D.size(), f) != D.size() || std::fread(N.data(), sizeof(double), 80, f) != 80 ||
      std::fread(P.data(), sizeof(double), P.size(), f) != P.size())
    return 4;
  std::fclose(f);
  const double den2 = (double)den * den, wide = std::ldexp(den2, -kFxDenBits), unwide = std::ldexp(1.0 / den2, kFxDenBits);
  auto d_at = [&](int c, int q, int r, int s) { return D[225 * (size_t)c + (3 * r + q / 3) * 15 + 3 * s + q % 3]; };
  std::vector<unsigned> ex((size_t)9 * nc);
  int eb[9] = {}, most[9];
  for (int q = 0; q < 9; q++) most[q] = kFxRaw;
  for (int c = 0; c < nc; c++) {
    int fd[9] = {}, load[3] = {}, all = 0;
    for (int q = 0; q < 9; q++) {
      for (int k = 0; k < 25; k++) fd[q] = std::max(fd[q], fx_exponent(d_at(c, q, k / 5, k % 5)));
      all = std::max(all, fd[q]);
    }
    for (int k = 0; k < 9; k++) load[k % 3] = std::max(load[k % 3], fx_exponent(P[9 * (size_t)c + k]));
    for (int q = 0; q < 9; q++) {
      const unsigned x = fx_pack(fd[q], q % 4 ? load[3 - q / 3 - q % 3] : 0, all);
      ex[9 * (size_t)c + q] = x;
      eb[q] = std::max(eb[q], fx_row_exp(x));
      most[q] = std::min(most[q], fx_most_exp(x));
    }
  }
  std::vector<long long> bound(nblk, 0);
  int cs[16];
  for (int b = 0; b < 16; b++) {
    double col[5];
    for (int r = 0; r < 5; r++) col[r] = N[16 * r + b];
    cs[b] = fx_column_sum(col);
  }
  auto corner = [](int b) { return b < 3; };
  for (int c = 0; c < nc; c++)
    for (int b = 0; b < nen; b++)
      bound[tgt[16 * c + b]] += (long long)cs[a[c]] * cs[b] + (corner(a[c]) && corner(b) ? 64 * 64 : 0);
  long long largest = 0;
  for (long long v : bound) largest = std::max(largest, v);
  const int grow = fx_growth(largest);
  double in_integers = 1.0;
  for (int q = 0; q < 9; q++)
    if (eb[q] + grow > most[q]) in_integers = 0.0;
  std::vector<long long> acc((size_t)9 * nblk, 0);
  std::vector<double> accw(acc.size(), 0.0);
  for (int c = 0; c < nc; c++) {
    for (int q = 0; q < 9; q++) {
      const int ee = fx_d_exp(ex[9 * (size_t)c + q]);
      Fx w[5], ww[5];
      for (int s = 0; s < 5; s++) {
        FxSum<62> sum;
        for (int r = 0; r < 5; r++) sum.add(fx_table(N[16 * r + a[c]], den), fx_split(fx_from_double(d_at(c, q, r, s), ee)));
        ww[s] = fx_split(sum.value());
        w[s] = fx_split(fx_shift(sum.value(), eb[q] + grow - ee));
      }
      for (int b = 0; b < nen; b++) {
        Fx n[5];
        for (int s = 0; s < 5; s++) n[s] = fx_table(N[16 * s + b], den);
        const size_t t = 9 * (size_t)tgt[16 * c + b] + q;
        acc[t] += fx_entry(n, w);
        accw[t] += fx_wide(fx_entry(n, ww), ee);
      }
    }
    if (!corner(a[c])) continue;
    for (int k = 0; k < 3; k++)
      for (int d = 0; d < 3; d++) {
        const double v = P[9 * (size_t)c + 3 * k + d];
        const int qm = d == 0 ? 5 : d == 1 ? 6 : 1, qp = d == 0 ? 7 : d == 1 ? 2 : 3;
        const size_t t = 9 * (size_t)tgt[16 * c + k];
        acc[t + qm] -= fx_load(v * den2, eb[qm] + grow);
        acc[t + qp] += fx_load(v * den2, eb[qp] + grow);
        accw[t + qm] -= v * wide;
        accw[t + qp] += v * wide;
      }
  }
  std::vector<double> hi(acc.size()), lo(acc.size());
  for (size_t t = 0; t < acc.size(); t++) {
    hi[t] = (double)(acc[t] >> 32);
    lo[t] = (double)(acc[t] & 0xffffffffll);
    accw[t] *= unwide;
  }
  FILE *g = std::fopen(argv[2], "wb");
  if (!g) return 6;
  const double g2 = grow;
  std::fwrite(&in_integers, sizeof(double), 1, g);
  std::fwrite(&g2, sizeof(double), 1, g);
  for (int q = 0; q < 9; q++) { const double e = eb[q] - 1022; std::fwrite(&e, sizeof(double), 1, g); }
  std::fwrite(hi.data(), sizeof(double), hi.size(), g);
  std::fwrite(lo.data(), sizeof(double), lo.size(), g);
  std::fwrite(accw.data(), sizeof(double), accw.size(), g);
  std::fclose(g);
  return 0;
}
