// The reciprocal of the fast variants' hot loops.
#ifndef JB_RCP_CUH
#define JB_RCP_CUH

// 1 / x of a float64 x whose size and reciprocal are normal numbers: the
// hardware's approximate reciprocal refined by one third-order step of the
// Newton family, r (1 + e + e^2) with e = 1 - x r (measured: e below 1e-6, so
// the step's error e^3 is below half an ulp; the result within 2 ulp).  No
// range fix-up and no branch, so that several of them interleave.  0 and
// infinity give NaN.
__device__ __forceinline__ double rcp_nr(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

#endif  // JB_RCP_CUH
