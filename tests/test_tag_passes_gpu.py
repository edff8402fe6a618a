"""The tagging passes at the edges of their launch shapes: extents around
the 32 x 8 cells of a block and the 32 cells a warp fills at a time, bodies
that cross several of them, lines without a band cell, and a second tagging
after the body has moved.  The masks are
whole numbers and must equal the oracle's."""
import numpy as np
import pytest

from feicar_b200 import fg, synth
import oracle as O

pytestmark = pytest.mark.gpu


def _oracle_masks(grid, body):
    oc = O.OracleCase(grid)
    oc.add_body(body)
    oc.set_iblank()
    solid = np.array(oc.field(0))
    assert oc.gcm(2.0, 2.0) == 0
    return solid, [np.array(oc.field(q)) for q in range(3)]


@pytest.mark.parametrize("at", [0.35, 0.8])
@pytest.mark.parametrize("cells", [(31, 17, 18), (32, 16, 16), (33, 15, 24), (65, 25, 17), (97, 18, 33)])
def test_masks(cells, at):
    h = 1.0 / min(cells)
    grid = synth.Grid(*[synth.uniform_nodes(n, 0, n * h) for n in cells])
    bodies = [synth.sphere_body((f * cells[0] * h, 0.5 * cells[1] * h, 0.5 * cells[2] * h), 0.5, 3)
              for f in (at, at - 0.07)]
    c = fg.Case(grid, fg.default_config())
    c.add_body(bodies[0])
    for n, body in enumerate(bodies):
        if n:
            c.update_body(0, body.verts)
        solid = c.set_iblank_body_fast()
        masks = c.gcm_set_internal_boundary()
        want, wants = _oracle_masks(grid, body)
        assert np.array_equal(solid, want)
        for got, w in zip(masks, wants):
            assert np.array_equal(got, w)
    c.close()
