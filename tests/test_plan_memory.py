"""Device memory of plan creation, on a fake CUDA runtime with a memory of a given size.

A plan fits where its own arrays fit: the buffer that its uploads go through is given back
before the later arrays are allocated, and where it is not to be had the uploads go row by
row, with the same contents.  Every upload is ordered by the plan's stream.
"""
import pytest

from tests.fake_cuda import FAKE_CUDA, FLAGS, SOURCES
from tests.host_cc import run_cpp

CODE = FAKE_CUDA + r"""
using namespace rsgpu;

template <typename P>
static int make(P &p, const rsgpu_config &c, std::vector<rsgpu_shot> &s, std::vector<unsigned char> &image)
{
    padded = by_rows = unordered = 0;
    const int st = p.create(&c, (int)s.size(), s.data());
    if (st == RSGPU_OK) image.assign((unsigned char *)p.arena, (unsigned char *)p.arena + p.arena_bytes);
    return st;
}

// Unlimited, then in a memory of just the plan's own arrays: status, uploads of each kind, same contents.
template <typename P>
static void both(const char *name, rsgpu_config c, int ns, int nx, int ny, int nz, bool adjoint)
{
    const int l = c.lpml;
    const size_t n = (size_t)(nx + 2 * l) * (ny ? ny + 2 * l : 1) * (nz + 2 * l);
    std::mt19937 rng(1);
    std::vector<std::vector<float>> par(8, std::vector<float>(n));
    for (auto &v : par) for (auto &x : v) x = rng() / 4.0e9f;
    std::vector<rsgpu_shot> s(ns);
    for (auto &q : s) {
        q.nx = nx; q.ny = ny; q.nz = nz;
        for (int k = 0; k < 8; k++) q.model[k] = par[k].data();
    }
    std::vector<unsigned char> a, b;
    size_t own = 0;
    capacity = ~size_t(0);
    {
        P p;
        p.adjoint_steps = adjoint;
        if (make(p, c, s, a) != RSGPU_OK) exit(1);
        own = used;
        printf("%s %d %d %d ", name, unordered, padded, by_rows);
    }
    if (used) exit(2);
    capacity = own;
    {
        P p;
        p.adjoint_steps = adjoint;
        const int st = make(p, c, s, b);
        printf("%d %d %d %d\n", st, padded, by_rows, (int)(a == b));
    }
    if (used) exit(3);
}

int main()
{
    rsgpu_config c{};
    c.precision = RSGPU_F32_FAST;
    c.order = 8; c.nt = 10;
    c.dx = c.dy = c.dz = 10.0; c.dt = 1e-3;
    c.tile = -1;
    c.lpml = 5;
    c.physics = RSGPU_ACOUSTIC2D;
    both<Plan>("a2", c, 50, 3, 0, 7, false);      // tables larger than the staging buffer
    both<Plan>("a2", c, 2, 160, 0, 145, false);
    c.physics = RSGPU_ELASTIC3D;
    both<Plan3D>("e3", c, 2, 20, 9, 11, true);    // work arrays behind the uploads
    c.physics = RSGPU_ACOUSTIC3D;
    both<Plan3D>("a3", c, 3, 20, 9, 11, false);
    c.physics = RSGPU_ELASTIC2D;
    for (c.launch_mode = 3; c.launch_mode <= 4; c.launch_mode++) both<Plan>("e2", c, 2, 160, 0, 145, false);
}
"""


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    out = run_cpp(tmp_path_factory.mktemp("plan_memory"), CODE, SOURCES, FLAGS)
    return [[w if k == 0 else int(w) for k, w in enumerate(row.split())] for row in out.splitlines()]


@pytest.mark.parametrize("row,uploads,staged", [(0, 150, True), (1, 6, False), (2, 16, True), (3, 12, False)])
def test_plan_fits_where_its_arrays_fit(lines, row, uploads, staged):
    # staged: the later arrays leave the room that the staging buffer needs before them
    _, _, padded, by_rows, status, padded2, by_rows2, same = lines[row]
    assert (padded, by_rows) == (uploads, 0)
    assert (status, same) == (0, 1)
    assert (padded2, by_rows2) == ((uploads, 0) if staged else (0, uploads))


def test_uploads_are_ordered_by_the_plans_stream(lines):
    assert len(lines) == 6 and all(status == 0 for _, _, _, _, status, *_ in lines)
    assert [unordered for _, unordered, *_ in lines] == [0] * 6
