"""Device memory of a Navier-Stokes grid: three state buffers, the host-order
copy and three words a cell for the viscous terms."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,word", [(0, 8), (1, 4)])
def test_the_viscous_terms_take_three_words_a_cell(cfsb, prec, word):
    import torch

    nx, ny = 3000, 2900
    kw = dict(precision=prec, rk=cfsb.RK_SSP3, hll=cfsb.HLL_DAVIS, bc=(cfsb.BC_PERIODIC,) * 4)
    cfsb.Solver(64, 64, viscous=cfsb.VISCOUS_NS, **kw).close()  # (the library's own allocations)
    used = {}
    for viscous in (cfsb.VISCOUS_OFF, cfsb.VISCOUS_NS):
        before = torch.cuda.mem_get_info()[0]
        with cfsb.Solver(nx, ny, viscous=viscous, **kw):
            used[viscous] = before - torch.cuda.mem_get_info()[0]
    terms = used[cfsb.VISCOUS_NS] - used[cfsb.VISCOUS_OFF]
    # (allocations come in blocks of 2 MiB)
    assert 0 < terms <= 3 * word * nx * ny + (4 << 20)
