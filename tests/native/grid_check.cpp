// grid_check.cpp -- TEST BUILD ONLY: the rule that tells which grids the FP64
// form takes as n dfq (phenom_acc.h), compiled for the host.
#include <cmath>

#include "../../gw_analysis_tools_gb300/csrc/phenom_acc.h"

using namespace gwt;

extern "C" {

// 1 where every frequency of a grid starting at bin n0 is on the line.
int gwr_on_line(const double *f, int n0, int N) {
  const double dfq = acc_spacing(f[N - 1], n0 + N - 1);
  for (int k = 0; k < N; k++)
    if (!acc_on_line(f[k], acc_off_line(f[k], n0 + k, dfq))) return 0;
  return 1;
}
// The rounding of a bin's frequency times t_c: error of its turns against long double.
double gwr_dev_error(double tc, float dev) {
  AccReq x;
  x.tc = (float)tc;
  const long double want = -(long double)x.tc * dev, got = (long double)(int64_t)acc_dev_turns(x, dev) / 18446744073709551616.0L;
  const long double e = got - want;
  return (double)fabsl(e - rintl(e));
}
}
