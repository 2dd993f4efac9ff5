// Host test shim: the table of roots of unity (simple3.0_b200/csrc/unit_root.h, the same source the library
// compiles).
#include "unit_root.h"

extern "C" void unit_roots(long long first, int count, long long n, double *cs)
{
    for (int i = 0; i < count; ++i) pftcc::unit_root(first + i, n, cs + 2 * i, cs + 2 * i + 1);
}
