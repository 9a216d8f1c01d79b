"""Rows that the engine applies a block each (256 columns and wider): the
persistent step against the grouped kernels, to the bit."""
import pytest

pytestmark = pytest.mark.gpu

# odd and even rows with and without a remainder of 32 columns; empty up lists, lists
# of one sign or shorter than four, full ones with every remainder
ROWS = [((11,), 0, 4), ((11,), 1, 5), ((11,), 11, 5), ((13,), 2, 4), ((11,), 5, 4), ((3, 4), 3, 6),
        ((13,), 3, 5), ((2, 2, 3), 4, 5)]


@pytest.mark.parametrize("dims,nu,nd", ROWS)
def test_persistent_rows_keep_the_grouped_bits(mb, cuda, dims, nu, nd):
    d = mb.sector(dims, nu, nd, 1.0, 4.0)
    kw = dict(seeds=[3], kmax=40, autotune=False, fused_threshold=1 << 62)
    a, b = (mb.batch_ground_states([d], persistent=p, **kw)[0] for p in (True, False))
    assert (a.e0, a.e0_raw, a.steps) == (b.e0, b.e0_raw, b.steps)
    dos = []
    for p in (True, False):
        eng = mb.Engine()
        eng.set_shape(persistent=p)
        eng.set_fused_threshold(1 << 62)
        rid = eng.try_submit_dos(d, n_moments=24, n_probes=1, seed=9)
        while eng.step(4):
            pass
        dos.append(eng.poll_dos(rid))
    assert dos[0][1:3] == dos[1][1:3] and (dos[0][0] == dos[1][0]).all()
