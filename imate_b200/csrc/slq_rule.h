// Which kernel serves an operator product that was not tuned.  Host code without
// CUDA, so that tests compile it alone.

#ifndef SLQ_RULE_H_
#define SLQ_RULE_H_

#include <algorithm>
#include <cstdint>

namespace slq {

// kinds of product kernels, as slq_tune_result reports them
enum { CAND_CSR = 0, CAND_RG = 1, CAND_TMA = 2, CAND_TC = 3, CAND_BLK = 4 };

// rpw (CAND_RG): rows of a group per warp (k_spmm_rg), 0 whole groups
// (k_spmm_rgs)
struct SpmmRule {
    int kind, rpw;
};

// The product of an operator without a block format and without a tuned
// choice, by rows, entries per row, group width (0: no groups) and block
// width: CSR, parts of row groups, whole row groups (b = 32 or 64, groups of 4
// or 8) or the TMA form (b = 128 or 256, groups of 16; only with a tensor map
// of the probe block, which slq_operator_dot and the second product of the
// normal equations do not have).  Measured on
// correlation matrices inside Krylov runs, whose passes over the basis leave
// L2 to the basis, us per product (n x entries per row, b: CSR / parts / whole
// groups):
//   FP64, 8 rows  12,000 x 40, 32: 18 / 44 / 34;  16,400 x 59, 32: 29 / 26 /
//                 23, 64: 37 / 32 / 27;  24,000 x 31, 32: 23 / 21 / 25, 64: 31
//                 / 33 / 30;  40,009 x 60, 64: 81 / 101 / 55;  65,537 x 31, 32:
//                 48 / 62 / 45;  200,000 x 61, 64: 366 / 372 / 223;  300,000 x
//                 26, 32: 158 / 162 / 150
//   FP64, 4 rows  12,000 x 40, 64: 23 / 31 / 28;  16,400 x 59, 64: 38 / 35 /
//                 26;  100,000 x 41, 64: 133 / 103 / 93;  300,000 x 26, 32: 157
//                 / 126 / 155, 64: 250 / 198 / 184
//   FP32, 8 rows  8,000 x 30, 256: 25 / 37;  16,400 x 59, 32: 20 / 23 / 17, 64:
//                 27 / 23 / 25, 128: 35 / 28;  24,000 x 31, 32: 17 / 19 / 19;
//                 32,768 x 98, 32: 44 / 48 / 36;  65,537 x 60, 32: 48 / 45 /
//                 46, 64: 76 / 66 / 78, 256: 208 / 152
//   FP32, 4 rows  16,400 x 59, 32: 20 / 24 / 19, 64: 27 / 23 / 21;  24,000 x 31,
//                 32: 17 / 20 / 18, 64: 21 / 20 / 19;  32,768 x 98, 64: 63 / 54
//                 / 43;  100,000 x 41, 32: 52 / 46 / 56, 64: 77 / 69 / 65;
//                 150,000 x 31, 64: 89 / 76 / 80
//   FP32, 16 rows (CSR / parts / TMA)  32,768 x 98, 256: 173 / 188 / 202;
//                 50,000 x 60, 128: 92 / 88 / 107, 256: 163 / 154 / 163;
//                 65,537 x 60, 128: 121 / 120 / 133, 256: 208 / 214 / 198;
//                 80,000 x 99, 128: 222 / 238 / 205;  150,000 x 60, 128: 253 /
//                 265 / 237;  220,000 x 60, 32: 136 / 151, 64: 234 / 215
//   the same, no tensor map  100,003 x 90, 256: 432 / 404;  150,000 x 31, 256:
//                 227 / 288;  220,000 x 61, 128: 354 / 322, 256: 748 / 626;
//                 262,144 x 149, 128: 1,124 / 748, 256: 2,487 / 1,408
// Small matrices have too few groups to hide a gather's latency.
inline SpmmRule spmm_rule(bool f64, int64_t rows, double per_row, int G, int b,
                          bool have_map)
{
    const SpmmRule csr{CAND_CSR, 0}, parts{CAND_RG, std::min(G, 8)}, whole{CAND_RG, 0};
    if (!G || rows < 16384 || b < 32 || b > 256) return csr;
    const bool long_rows = per_row >= 48.0;
    if (f64)
    {
        if (b > 64 || G > 8) return csr;
        return (G == 4 || long_rows || rows >= 32768) ? whole : csr;
    }
    if (G == 16)
    {
        if (b >= 128 && have_map)
            return rows >= (b == 128 ? 73728 : 49152) ? SpmmRule{CAND_TMA, 0} : csr;
        return rows >= 200000 ? parts : csr;
    }
    if (b == 32 && long_rows && rows < (G == 4 ? 98304 : 65536)) return whole;
    if (b == 64 && G == 4 && rows < 131072) return whole;
    return (b >= 128 || rows >= 65536) ? parts : csr;
}

}  // namespace slq

#endif  // SLQ_RULE_H_
