// Host entry points over polysplat_gb300/csrc/ndc.h, built by tests/test_ndc.py.
#include "../polysplat_gb300/csrc/ndc.h"

extern "C" void ndc_both(int n, const float* v, int S, float* fast, float* ref)
{
    for (int i = 0; i < n; i++) {
        fast[i] = gsr_ndc::to_pix(v[i], S);
        ref[i] = gsr_ndc::to_pix_double(v[i], S);
    }
}
