// div.h -- division by a value that many quotients share.
#pragma once
#include "hd.h"

namespace irbc {

// x / y for a divisor whose correctly rounded reciprocal r is at hand, rounded
// as the division is (P. Markstein, IBM J. Res. Dev. 34 (1990) 111: from a
// quotient within one ulp, q + (x - q y) r is the correctly rounded one; the
// first correction brings it there).  Five dependent operations and no branch,
// where a division takes about 150 cycles.  The residuals x - q y have to be
// representable: equal to the division for |x| from 2^-969 on, a divisor whose
// reciprocal is normal, and a quotient that is.  Below that the last bit may
// differ; zeros lose their sign, and infinities and what overflows become NaN.
struct Divisor {
  double y, r;
};
IRBC_HD double div_by(double x, Divisor d) {
  double q = x * d.r;
  q = fma(fma(-d.y, q, x), d.r, q);
  return fma(fma(-d.y, q, x), d.r, q);
}
IRBC_HD double div3(double x) { return div_by(x, Divisor{3.0, 1.0 / 3.0}); }

}  // namespace irbc
