// The grid cell of a mesh triangle (pg_ttfilter.cuh): in range whatever the
// coordinate, the floor of the quotient inside the grid.
#include <cmath>
#include <cstdio>
#include <initializer_list>
#include <limits>
#include "../parmec_gb300/csrc/pg_ttfilter.cuh"

int main()
{
  long bad = 0, n = 0;
  const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
  for (const int dim : {1, 2, 5, 512, 1 << 20})
    for (const double h : {1e-3, 1.0, 1e6})
      for (const double org : {0.0, -2.5, 3e5})
      {
        for (const double x : {nan, -nan, inf, -inf, 1e308, -1e308, 1e-320, 0.0, -0.0})
        {
          const int c = pgtf::grid_cell(x, org, h, dim);
          bad += c < 0 || c >= dim || (x != x && c != 0);
          n ++;
        }
        for (int k = -3; k < 4 * dim && k < 1000; k ++)
        {
          const double x = org + h * (0.25 * k), q = std::floor((x - org) / h);
          const int want = q < 0.0 ? 0 : q > dim - 1 ? dim - 1 : (int)q;
          bad += pgtf::grid_cell(x, org, h, dim) != want;
          n ++;
        }
      }
  bad += pgtf::grid_cell(1.0, nan, 1.0, 4) != 0;
  printf("%ld %ld\n", bad, n);
  return 0;
}
