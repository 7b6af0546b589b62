"""The exact kernels' division by a spacing equals the host's division, bit for bit.

The same header that the kernels include, compiled for the host: zeros of both signs,
subnormals, infinities and NaN, operands beside the switch to the double quotient, divisors
that fail the formula's check, each alone and as the neighbour of an operand of the other path.
"""
from tests.host_cc import run_cpp

CODE = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <limits>
#include "exact_div.cuh"
#include "rsgpu_host.h"
using namespace rsgpu;
static float of(unsigned u) { float f; std::memcpy(&f, &u, 4); return f; }
static bool same(float a, float b) { return std::isnan(a) ? std::isnan(b) : bits_of(a) == bits_of(b); }
int main()
{
    const float inf = std::numeric_limits<float>::infinity();
    int failed = 0;
    // 9.00014782 and 5.99992752 fail the check; the last ones are out of its range
    for (float d : {10.f, 8.f, 16.f, 12.5f, 7.3f, 5.f, 6.25f, 0.01f, 9.00014782f, 5.99992752f, 333.3f, 1e-20f, 3e30f}) {
        const Rcp<float> r = divisor(d);
        failed += r.lo == 0xffffffffu;
        auto check = [&](float x) {
            const volatile float want = x / d;
            if (!same(div_by(x, d, r), want)) { printf("%a / %a = %a, not %a\n", x, d, want, div_by(x, d, r)); return false; }
            // beside a tiny operand, an ordinary one, a zero
            float v[4] = {x, 1e-41f, -0.0f, 3.7f};
            const volatile float w[4] = {v[0] / d, v[1] / d, v[2] / d, v[3] / d};
            div_by4(v, d, r);
            for (int j = 0; j < 4; j++)
                if (!same(v[j], w[j])) { printf("lane %d: %a, not %a (%a / %a)\n", j, v[j], w[j], x, d); return false; }
            return true;
        };
        for (float x : {0.f, -0.f, inf, -inf, std::nanf(""), of(1), of(0x80000001u), of(0x7f7fffffu), of(0xff7fffffu)})
            if (!check(x)) return 1;
        if (r.lo != 0xffffffffu)                    // operands around the switch
            for (unsigned b = (r.lo + 1) / 2 - 300; b < (r.lo + 1) / 2 + 300; b++)
                if (!check(of(b)) || !check(of(b | 0x80000000u))) return 1;
        for (unsigned long long b = 0; b < (1ull << 32); b += 4099)
            if (!check(of((unsigned)b))) return 1;
    }
    printf("%d\n", failed);
}
"""


def test_division_equals_the_hosts(tmp_path):
    failed = int(run_cpp(tmp_path, CODE, ["host_prep.cpp"], ["-O2", "-Wl,--unresolved-symbols=ignore-all", "-no-pie"]))
    assert 3 <= failed <= 4
