"""Split of the 3D correlations over a launch: every plane once, within a grid's limit in z."""
from tests.host_cc import run_cpp

CODE = r"""
#include <cstdio>
#include "rsgpu_adjoint.h"
int main()
{
    const int shots[] = {1, 2, 7, 100, 524, 525, 2427, 5041, 5042, 9000, 32767, 32768, 65534, 65535};
    const int planes[] = {1, 2, 7, 8, 9, 16, 101, 104, 1000, 4097};
    for (int n : shots)
        for (int z : planes) {
            const rsgpu::CorrChunks c = rsgpu::corr_chunks(n, z);
            if ((long long)n * c.count > 65535) { printf("%d shots of %d planes: %d chunks\n", n, z, c.count); return 1; }
            // the last chunk holds a plane, and the chunks hold all of them
            if ((c.count - 1) * c.planes >= z || (long long)c.count * c.planes < z) { printf("%d %d\n", n, z); return 2; }
            // no longer than need be
            if (c.planes != 8 && (long long)n * ((z + c.planes - 2) / (c.planes - 1)) <= 65535) { printf("%d %d\n", n, z); return 3; }
            if (n < 100 && c.planes != 8) return 4;
        }
}
"""


def test_corr_chunks(tmp_path):
    run_cpp(tmp_path, CODE)
