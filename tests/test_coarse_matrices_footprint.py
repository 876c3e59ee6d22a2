"""Which coarsest levels hold the matrices of their lines (dense_pays,
csrc/tpls_modes.cuh): lines of up to 64 points whatever their size, none above.
A level of 63 points a line has fewer cells than one of 65, so the larger
footprint, and on the GPU the larger context, shows its matrices."""
import pytest

GRIDS = [(25, 75), (35, 75), (69, 141)]  # matrices of 16, 22 and 81 MB


def _footprint(nx, ny, nz):
    from tpls_gb300.serve import GpuBackend
    return GpuBackend().lib.tpls_footprint_bytes(nx, ny, nz, 0)


@pytest.mark.parametrize("ny,nz", GRIDS)
def test_footprint_counts_them_up_to_64_points(ny, nz):
    """Without matrices the footprint does not fall with the cells; those of 63
    points outweigh the two points a line that they have fewer."""
    at63, at65, at67 = (_footprint(nx, ny, nz) for nx in (63, 65, 67))
    assert at63 > at65
    assert at67 >= at65


@pytest.mark.gpu
@pytest.mark.parametrize("ny,nz", GRIDS)
def test_context_allocates_them_as_counted(ny, nz):
    import torch
    from tpls_gb300.api import TplsGpu
    from tpls_gb300.channel import make_case
    used = []
    for nx in (63, 65):
        p, uin, _ = make_case("A", nx=nx, ny=ny, nz=nz)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        with TplsGpu(nx, ny, nz, p, uin) as g:
            g.sync()
            used.append(free - torch.cuda.mem_get_info()[0])
    assert used[0] > used[1]
