// Implicit QL with shifts on a symmetric tridiagonal matrix, tracking only
// the first row of the eigenvector matrix (Golub-Welsch: the FTLM weights are
// the squared first components), then an ascending insertion sort. A warp per
// matrix in the engine's batched Ritz stage (lanczos.cu), a thread per matrix in
// the allocation-free entry point (noalloc.cu).
#pragma once

namespace ftlm {

// Rotation of (f, g) onto its norm: rr = |(f, g)|, s = f / rr, c = g / rr; rr = 0 for
// a zero vector. The squares are used as they are where they neither overflow nor
// lose bits to underflow, and everything comes from one reciprocal root h: a Newton
// step corrects rr = r2 h by its residual r2 - rr^2, and each quotient q = f h by
// f - q rr (Markstein's correction), so that all three are rounded about once, as
// hypot (2 ulp) and two divisions gave them. Without the residuals they are 1 to 2 ulp off
// and the eigenvalues' root-mean-square error on tridiagonals of 20 to 120 steps is
// 15% larger. The rotation is most of the sweep's dependent chain (5 x 80 steps: 2.8 ms
// with hypot and divisions, 2.0 with a root and divisions, 1.1 this way, 1.0 without
// the residuals).
__device__ __forceinline__ void ql_rotation(double f, double g, double& rr, double& s, double& c) {
  const double r2 = fma(f, f, g * g);
  if (r2 > 1e-200 && r2 < 1e200) {
    const double h = rsqrt(r2), r0 = r2 * h, sf = f * h, cg = g * h;
    rr = fma(0.5 * h, fma(-r0, r0, r2), r0);
    s = fma(h, fma(-sf, rr, f), sf);
    c = fma(h, fma(-cg, rr, g), cg);
  } else {
    rr = hypot(f, g);
    s = f / rr;
    c = g / rr;
  }
}

// d[0..n): diagonal, e[0..n-1): off-diagonal (e[n-1] = 0), z: first row of
// the eigenvector matrix (1, 0, ..., 0 on entry). A is any indexable view of
// doubles. Returns false when an eigenvalue needed more than 200 iterations.
// WARP: called by all 32 lanes with the same arrays. The lanes look for the next
// negligible off-diagonal 32 at a time; the sweeps and the sort, which read what
// they have just written, run on lane 0 alone, and a __syncwarp stands between
// every store and the other lanes' next loads (all lanes in step is not promised).
template <bool WARP = false, typename A>
__device__ __forceinline__ bool ql_first_row(int n, A d, A z, A e) {
  bool ok = true;
  const double eps = 2.220446049250313e-16;
  const bool lead = !WARP || (threadIdx.x & 31) == 0;
  for (int l = 0; l < n; ++l) {
    int iter = 0;
    while (true) {
      int m = l;
      if constexpr (WARP) {
        const int lane = threadIdx.x & 31;
        unsigned int hit = 0;
        for (; !hit && m < n - 1; m += 32) {
          const int k = m + lane;
          hit = __ballot_sync(0xffffffffu, k < n - 1 && fabs(e[k]) <= eps * (fabs(d[k]) + fabs(d[k + 1])));
        }
        m = hit ? m - 32 + __ffs(hit) - 1 : n - 1;
      } else {
        for (; m < n - 1; ++m) {
          const double dd = fabs(d[m]) + fabs(d[m + 1]);
          if (fabs(e[m]) <= eps * dd) break;
        }
      }
      if (m == l) break;
      if (++iter > 200) {
        ok = false;
        break;
      }
      if constexpr (WARP) __syncwarp();  // every lane has loaded
      if (lead) {
        double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
        double rr = hypot(g, 1.0);
        double dm = d[m];  // d[i + 1]
        g = dm - d[l] + e[l] / (g + copysign(rr, g));
        double s = 1.0, c = 1.0, p = 0.0, zm = z[m];  // zm: z[i + 1]
        double en = e[m - 1], dn = d[m - 1], zn = z[m - 1];  // row i's, loaded one rotation ahead
        bool underflow = false;
        for (int i = m - 1; i >= l; --i) {
          const double ei = en, di = dn, zi = zn;
          if (i > l) {
            en = e[i - 1];
            dn = d[i - 1];
            zn = z[i - 1];
          }
          const double f = s * ei, b = c * ei;
          double sn, cn;
          ql_rotation(f, g, rr, sn, cn);
          e[i + 1] = rr;
          if (rr == 0.0) {
            d[i + 1] = dm - p;
            z[i + 1] = zm;
            e[m] = 0.0;
            underflow = true;
            break;
          }
          s = sn;
          c = cn;
          g = dm - p;
          rr = (di - g) * s + 2.0 * c * b;
          p = s * rr;
          d[i + 1] = g + p;
          g = c * rr - b;
          z[i + 1] = s * zi + c * zm;
          zm = c * zi - s * zm;
          dm = di;
        }
        if (!underflow) {
          d[l] = dm - p;
          z[l] = zm;
          e[l] = g;
          e[m] = 0.0;
        }
      }
      if constexpr (WARP) __syncwarp();
    }
  }
  if constexpr (WARP) __syncwarp();
  if (lead) {
    for (int i = 1; i < n; ++i) {  // insertion sort, ascending
      const double dk = d[i], zk = z[i];
      int j = i - 1;
      while (j >= 0 && d[j] > dk) {
        d[j + 1] = d[j];
        z[j + 1] = z[j];
        --j;
      }
      d[j + 1] = dk;
      z[j + 1] = zk;
    }
  }
  if constexpr (WARP) __syncwarp();
  return ok;
}

}  // namespace ftlm
