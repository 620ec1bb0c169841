// The truncation rules on the device, shared by the single and the batched factorisations.
#pragma once
#include <cstdint>

// ============================================================== truncation
// By one thread, which walks the spectrum in the same sequential order as the CPU
// rules it restates, so both give bit-identical sums.  n <= 2*chi is a few
// thousand values: tens of microseconds, once per bond.
__device__ inline void truncate_spectrum(const double* P, int64_t n, int64_t maxdim,
                                         int64_t mindim, double cutoff, int absoluteCutoff, int doRelCutoff,
                                         int legacy, double* out) {
  const int64_t origm = n;
  double truncerr = 0.0, docut = 0.0;
  int64_t keep = 1;
  if (origm == 0) {
    out[0] = 0; out[1] = 0; out[2] = 0;
    return;
  }
  if (maxdim <= 0 || maxdim > origm) maxdim = origm;
  if (!legacy) {
    // ITensors (NDTensors) CPU rule: cumulative discarded weight.
    if (origm == 1) {
      out[0] = 1; out[1] = 0.0; out[2] = fabs(P[0]) / 2;
      return;
    }
    const double sgn = (P[0] < 0.0) ? -1.0 : 1.0;
    // trailing negative weights count as zero
    int64_t lastpos = origm;  // values at index >= lastpos are treated as 0
    for (int64_t i = origm - 1; i >= 0; --i) {
      if (sgn * P[i] >= 0.0) break;
      lastpos = i;
    }
#define PV(i) ((i) >= lastpos ? 0.0 : sgn * P[(i)])
    if (mindim < 1) mindim = 1;
    int64_t nn = origm;
    while (nn > maxdim) { truncerr += PV(nn - 1); nn--; }
    if (absoluteCutoff) {
      while (PV(nn - 1) <= cutoff && nn > mindim) { truncerr += PV(nn - 1); nn--; }
    } else {
      double scale = 1.0;
      if (doRelCutoff) {
        scale = 0.0;
        for (int64_t i = 0; i < origm; ++i) scale += PV(i);
        if (scale == 0.0) scale = 1.0;
      }
      const double thr = __dmul_rn(cutoff, scale);
      while ((__dadd_rn(truncerr, PV(nn - 1)) <= thr) && nn > mindim) {
        truncerr += PV(nn - 1);
        nn--;
      }
      truncerr /= scale;
    }
    if (nn < 1) nn = 1;
    if (nn < origm) {
      docut = (PV(nn - 1) + PV(nn)) / 2;
      if (fabs(PV(nn - 1) - PV(nn)) < __dmul_rn(1e-3, PV(nn - 1)))
        docut = __dadd_rn(docut, __dmul_rn(1e-3, PV(nn - 1)));
    }
#undef PV
    keep = nn;
  } else {
    // src/tensor/cutruncate.jl:1-93, step by step.
    if (mindim < 1) mindim = 1;
    if (mindim > maxdim) mindim = maxdim;
    double maxP = P[0];
    for (int64_t i = 1; i < origm; ++i) maxP = fmax(maxP, P[i]);
    if (maxP == 0.0) {
      out[0] = 1; out[1] = 0.0; out[2] = 0.0;
      return;
    }
    if (origm == 1) {
      out[0] = 1; out[1] = 0.0; out[2] = maxP / 2;
      return;
    }
#define RP(i) (signbit(P[(i)]) ? 0.0 : P[(i)])
    int64_t nn = origm;
    if (nn > maxdim) {
      for (int64_t i = 0; i < nn - maxdim; ++i) truncerr += RP(i);  // head sum, as written
      nn = maxdim;
    }
    // cut_ind: first index whose value is strictly below the threshold
    // (cuBLAS iamax over the +-2/0 flag vector), 0 when there is none.
    int64_t cut_ind = 0;
    if (absoluteCutoff) {
      for (int64_t i = 0; i < origm; ++i)
        if (RP(i) - cutoff < 0.0) { cut_ind = i; break; }
      nn = min(maxdim, origm - cut_ind);
      nn = max(nn, mindim);
      for (int64_t i = cut_ind; i < origm; ++i) truncerr += RP(i);
    } else {
      double scale = 1.0;
      if (doRelCutoff) {
        scale = 0.0;
        for (int64_t i = 0; i < origm; ++i) scale += P[i];
        scale = scale > 0.0 ? scale : 1.0;
      }
      for (int64_t i = 0; i < origm; ++i)
        if (__dsub_rn(__dadd_rn(RP(i), truncerr), __dmul_rn(cutoff, scale)) < 0.0) { cut_ind = i; break; }
      if (cut_ind > 0) {
        for (int64_t i = cut_ind; i < origm; ++i) truncerr += RP(i);
      } else {
        for (int64_t i = 0; i < maxdim; ++i) truncerr += RP(i);
      }
      nn = min(maxdim, origm - cut_ind);
      nn = max(nn, mindim);
      truncerr = (scale == 0.0) ? 0.0 : truncerr / scale;
    }
#undef RP
    if (nn < 1) nn = 1;
    if (nn < origm) {
      docut = (P[nn - 1] + P[nn]) / 2;
      if (fabs(P[nn - 1] - P[nn]) < __dmul_rn(1e-3, P[nn - 1]))
        docut = __dadd_rn(docut, __dmul_rn(1e-3, P[nn - 1]));
    }
    keep = nn;
  }
  out[0] = (double)keep;
  out[1] = truncerr;
  out[2] = docut;
}
