// divide.hpp -- several divisions by one number, with its reciprocal formed once.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define BM4DOF_HD __host__ __device__ __forceinline__
#else
#define BM4DOF_HD inline
#endif

namespace bm4dof {

// a / b for finite a, rounded as the division rounds it (but 0 for a =
// -0), with y = 1 / b correctly rounded.  In units of the last place of q = a y
// rounded, m(x) being the mantissa of x in [1, 2):
//
//   * a / b is at most 1/2 + m(q) m(b) / 4 from q: q's own rounding and y's.
//   * Up to 1: Markstein's theorem (IBM J. Res. Dev. 34(1), 1990).  The remainder r =
//     a - b q is exact, and q + r y rounds to the quotient.
//   * From 1 to 3/2: the quotient is the neighbour of q on that side.  r may need a
//     25th bit, and its rounding and y's error move q + r y by less than 2^-22.4,
//     too little to reach 3/2 unless m(q) m(b) > 4 - 2^-20.4.  That leaves m(b) >= 2 - 3
//     2^-23 (and of these the odd ones, whose reciprocals lie near a tie): for them
//     every a has been compared with the division.
//
// The bounds keep all this clear of the subnormal numbers: q is at least 2^-120 and
// the remainder a multiple of 2^-146.  (With b up to 2^60 subnormal quotients came
// out wrong, three in a million next to a tie.)
BM4DOF_HD float divide_by(float a, float b, float y)
{
	if ((fabsf(a) < 0x1p-100f && a != 0.f) || !(b >= 1.f && b <= 0x1p20f)) return a / b;
	const float q = a * y;
	return fmaf(fmaf(-b, q, a), y, q);
}

}  // namespace bm4dof
