// tile_shim.cpp with quotients GSR_TT_ULPS units off the rounded ones, as far as
// the device's fast-math division may be (tests/test_tile_division.py).
#include <cmath>

inline float off_quotient(float a, float b)
{
    float q = a / b;
    for (int k = 0; k < (GSR_TT_ULPS < 0 ? -GSR_TT_ULPS : GSR_TT_ULPS); k++)
        q = std::nextafter(q, GSR_TT_ULPS < 0 ? -INFINITY : INFINITY);
    return q;
}
#define GSR_TT_DIV(a, b) off_quotient(a, b)
#include "tile_shim.cpp"
