"""Snapshots restore every cell from one place: blocks that overlapped would be written by
threads that race, with values that differ in 16-bit slots (each block has its own scale)."""
import pytest

from tests.fake_cuda import FAKE_CUDA, FLAGS, SOURCES
from tests.host_cc import run_cpp

CODE = FAKE_CUDA + r"""
#include "rsgpu_adjoint.h"
static size_t cells = 0, twice = 0, restores = 0;
namespace rsgpu {
size_t residual_partials(int) { return 1; }
cudaError_t launch_step_2d(int, int, int, int, int, const void *, const void *, const void *, int *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_injrec_2d(int, const void *, const void *, int, double, int, const int *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_corr_rtm_a2d(int, int, const void *, int, int, int, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ckpt_save(int, int, const CkptSeg *, int, int, void *, float *, unsigned *, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ckpt_load(int, int, const CkptSeg *segs, int nseg, int max_rows, const void *, const float *, cudaStream_t)
{
    std::map<char *, int> seen;
    for (int i = 0; i < nseg; i++)
        for (int r = 0; r < segs[i].rows; r++)
            for (int c = 0; c < segs[i].cols; c++) seen[(char *)segs[i].src + 4 * ((size_t)r * segs[i].pitch + c)]++;
    cells = seen.size();
    for (auto &s : seen) twice += s.second > 1;
    restores++;
    return cudaSuccess;
}
}

int main()
{
    for (int method : {RSGPU_SNAP_OPTIMAL, RSGPU_SNAP_FULL, RSGPU_SNAP_EDGES})
        for (auto n : {std::pair<int, int>{23, 14}, {1, 9}, {9, 1}}) {
            rsgpu_config c{};
            c.precision = RSGPU_F32_EXACT;
            c.physics = RSGPU_ACOUSTIC2D;
            c.order = 4; c.nt = 8; c.lpml = 5;
            c.dx = c.dz = 10.0; c.dt = 1e-3;
            c.tile = -1;
            rsgpu_adjoint_opts o{};
            o.ncheck = 3; o.ckpt_precision = RSGPU_CKPT_F16;
            o.nhx = o.nhz = 1;
            o.snapmethod = method; o.snapinc = 1;
            std::vector<float> par((size_t)(n.first + 10) * (n.second + 10), 1.0f), wav(c.nt), image((size_t)n.first * n.second);
            const int map[2] = {0, 0};
            const float shift[2] = {0.25f, 0.5f};
            rsgpu_adjoint_shot s{};
            s.shot.nx = n.first; s.shot.nz = n.second;
            for (int k = 0; k < 3; k++) s.shot.model[k] = par.data();
            s.shot.nsrc = s.shot.nrec = 1;
            s.shot.smap = s.shot.gmap = map;
            s.shot.sshift = s.shot.gshift = shift;
            s.shot.wavelet = wav.data();
            s.data = wav.data();
            s.image = image.data();
            restores = twice = 0;
            const rsgpu_status st = rsgpu_rtm_image(&c, &o, 1, &s);
            if (st != RSGPU_OK) { printf("status %d: %s\n", st, rsgpu_last_error()); return 1; }
            printf("%d %d %d %zu %zu %zu\n", method, n.first, n.second, restores, cells, twice);
        }
}
"""


def test_no_cell_is_restored_twice(tmp_path):
    out = run_cpp(tmp_path, CODE, SOURCES + ["adjoint.cpp", "adjoint3d.cpp", "revolve.cpp"], FLAGS)
    for method, nx, nz, restores, cells, twice in ([int(w) for w in line.split()] for line in out.splitlines()):
        assert restores > 0 and twice == 0, out
        if method == 2:          # two columns of the interior rows, two rows of the interior columns
            assert cells == 2 * nz + 2 * nx - 1
