// Implicit QL with Wilkinson shifts on a symmetric tridiagonal matrix, run by
// one warp.  In a file of its own, with nothing from CUDA but the warp
// primitives, so that tests compile it for the host and run the lanes of the
// warp in orders of their own.

#ifndef SLQ_QL_CUH_
#define SLQ_QL_CUH_

#include <cmath>

namespace slq {

// d (diagonal), e (off-diagonal) and z (first eigenvector entries) of k
// entries in shared memory.  Lane 0 alone walks the chain of rotations, reads
// and stores; the other lanes take part in the search for a negligible entry
// and wait at the end of a sweep, so nothing a lane reads is written
// meanwhile.  Returns 1 if an eigenvalue took more than 60 iterations.
template <typename A>
__device__ inline int ql_first_row(A d, A e, A z, int k, int lane)
{
    if (k <= 1) return 0;
    const double eps = 2.220446049250313e-16;
    for (int l = 0; l < k; ++l)
    {
        int iter = 0;
        for (;;)
        {
            // the first negligible off-diagonal entry from l on
            int mm = k - 1;
            for (int base = l; base < k - 1; base += 32)
            {
                const int i = base + lane;
                const bool small =
                    i < k - 1 && fabs(e[i]) <= eps * (fabs(d[i]) + fabs(d[i + 1]));
                const unsigned hit = __ballot_sync(0xffffffffu, small);
                if (hit)
                {
                    mm = base + __ffs(hit) - 1;
                    break;
                }
            }
            if (mm == l) break;
            if (++iter > 60) return 1;
            __syncwarp();  // every lane has read what the sweep overwrites
            if (lane == 0)
            {
                double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
                double r = fabs(g) < 1e150 ? sqrt(g * g + 1.0) : hypot(g, 1.0);
                g = d[mm] - d[l] + e[l] / (g + (g >= 0.0 ? r : -r));
                double s = 1.0, c = 1.0, p = 0.0;
                bool deflated = false;
                // zf and dh carry z[i + 1] and the old d[i + 1]; dn, en, zn
                // are the entries of the next rotation
                double zf = z[mm], dh = d[mm];
                double dn = d[mm - 1], en = e[mm - 1], zn = z[mm - 1];
                for (int i = mm - 1; i >= l; --i)
                {
                    const double di = dn, ei = en, zi = zn;
                    if (i > l)
                    {
                        dn = d[i - 1];
                        en = e[i - 1];
                        zn = z[i - 1];
                    }
                    const double f = s * ei;
                    const double bb = c * ei;
                    const double h = f * f + g * g;
                    if (h > 1e-280 && h < 1e280)
                    {
                        const double q = rsqrt(h);
                        r = h * q;
                        s = f * q;
                        c = g * q;
                    }
                    else
                    {
                        // squares that would leave the range of a double
                        r = hypot(f, g);
                        if (r == 0.0)
                        {
                            e[i + 1] = 0.0;
                            d[i + 1] = dh - p;
                            z[i + 1] = zf;
                            e[mm] = 0.0;
                            deflated = true;
                            break;
                        }
                        s = f / r;
                        c = g / r;
                    }
                    g = dh - p;
                    const double t = (di - g) * s + 2.0 * c * bb;
                    p = s * t;
                    e[i + 1] = r;
                    d[i + 1] = g + p;
                    z[i + 1] = s * zi + c * zf;
                    g = c * t - bb;
                    zf = c * zi - s * zf;
                    dh = di;
                }
                if (!deflated)
                {
                    d[l] = dh - p;
                    z[l] = zf;
                    e[l] = g;
                    e[mm] = 0.0;
                }
            }
            __syncwarp();
        }
    }
    return 0;
}

}  // namespace slq

#endif  // SLQ_QL_CUH_
