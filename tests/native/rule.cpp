#include "slq_rule.h"

// kind and rows per warp of the built-in choice
extern "C" void rule(int f64, long long rows, double per_row, int G, int b, int have_map,
                     int* out)
{
    const slq::SpmmRule r = slq::spmm_rule(f64 != 0, rows, per_row, G, b, have_map != 0);
    out[0] = r.kind;
    out[1] = r.rpw;
}
