/* Host driver of the fixed-point contraction (fx.cuh) for
   tests/test_fx_host.py: reads from argv[1] a row of nc contributions of one
   table (header: nc, nen, nblk, 1 for integer table values; per contribution the row slot a, the nen
   block targets and D 15x15; then the 5x16 table) and adds them up the way the row
   assembly does, in fixed point and in double, with the target blocks of
   every slot; writes both rows (9 nblk values each, block layout 9 t + q) to
   argv[2]. */
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
  int hdr[4];
  if (std::fread(hdr, sizeof(int), 4, f) != 4) return 4;
  const int nc = hdr[0], nen = hdr[1], nblk = hdr[2], den = 10000;
  const bool ints = hdr[3] != 0;
  std::vector<int> a(nc), tgt((size_t)nc * 16);
  std::vector<double> D((size_t)nc * 225), N(80);
  if (std::fread(a.data(), sizeof(int), nc, f) != (size_t)nc || std::fread(tgt.data(), sizeof(int), tgt.size(), f) != tgt.size() ||
      std::fread(D.data(), sizeof(double), D.size(), f) != D.size() || std::fread(N.data(), sizeof(double), 80, f) != 80)
    return 4;
  std::fclose(f);
  std::vector<double> kd((size_t)9 * nblk, 0.0), kx(kd.size());
  std::vector<long long> acc(kd.size(), 0);
  int eb[9] = {}, ebe[9];
  auto exps = [&](int c, int out[9]) {
    for (int q = 0; q < 9; q++) {
      out[q] = 0;
      for (int r = 0; r < 5; r++)
        for (int s = 0; s < 5; s++) {
          const int x = fx_exponent(D[225 * (size_t)c + (3 * r + q / 3) * 15 + 3 * s + q % 3]);
          out[q] = x > out[q] ? x : out[q];
        }
    }
  };
  for (int c = 0; c < nc; c++) {
    exps(c, ebe);
    for (int q = 0; q < 9; q++) eb[q] = ebe[q] > eb[q] ? ebe[q] : eb[q];
  }
  /* the largest block bound of the row */
  std::vector<long long> bound(nblk, 0);
  int cs[16];
  for (int b = 0; b < 16; b++) {
    double col[5];
    for (int r = 0; r < 5; r++) col[r] = N[16 * r + b];
    cs[b] = fx_column_sum(col);
  }
  for (int c = 0; c < nc; c++)
    for (int b = 0; b < nen; b++) bound[tgt[16 * c + b]] += (long long)cs[a[c]] * cs[b];
  long long most = 0;
  for (long long v : bound) most = v > most ? v : most;
  const int grow = fx_growth(most);
  for (int c = 0; c < nc; c++) {
    exps(c, ebe);
    const double *Dc = D.data() + 225 * (size_t)c;
    for (int q = 0; q < 9; q++) {
      Fx w[5];
      double wd[5];
      for (int s = 0; s < 5; s++) {
        FxSum<62> sum;
        FxIntSum<14> isum;
        double v = 0.0;
        for (int r = 0; r < 5; r++) {
          const double d = Dc[(3 * r + q / 3) * 15 + 3 * s + q % 3], n = N[16 * r + a[c]];
          const Fx x = fx_split(fx_from_double(d, ebe[q]));
          if (std::fabs(fx_to_double(x, ebe[q]) - d) > std::ldexp(1.0, ebe[q] - 1022 - 60)) return 5;
          if (ints) isum.add((int)llrint(n * den), x);
          else sum.add(fx_table(n, den), x);
          v = std::fma(n, d, v);
        }
        w[s] = fx_split(fx_shift(ints ? isum.value() : sum.value(), eb[q] + grow - ebe[q]));
        wd[s] = v;
      }
      for (int b = 0; b < nen; b++) {
        FxSum<63> sum;
        FxIntSum<15> isum;
        double *o = &kd[9 * (size_t)tgt[16 * c + b] + q];
        for (int s = 0; s < 5; s++) {
          if (ints) isum.add((int)llrint(N[16 * s + b] * den), w[s]);
          else sum.add(fx_table(N[16 * s + b], den), w[s]);
          *o = std::fma(N[16 * s + b], wd[s], *o);
        }
        acc[9 * (size_t)tgt[16 * c + b] + q] += ints ? isum.value() : sum.value();
      }
    }
  }
  const double g2 = grow;
  for (size_t t = 0; t < acc.size(); t++) kx[t] = (double)acc[t] * std::ldexp(1e-8, eb[t % 9] + grow - 1022 - kFxUnit);
  FILE *g = std::fopen(argv[2], "wb");
  if (!g) return 6;
  std::fwrite(&g2, sizeof(double), 1, g);
  std::fwrite(kx.data(), sizeof(double), kx.size(), g);
  std::fwrite(kd.data(), sizeof(double), kd.size(), g);
  std::fclose(g);
  return 0;
}
