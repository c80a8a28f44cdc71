"""The barotropic kernels' forms against each other on ragged and dry domains.

The resident form (1) picks a tile shape by the domain's size, and the
multi-tile form (2) skips the tiles without sea.  Both keep the operation
order of the generic form (3), so every field of the state is held to bit
equality with it (signed zeros are equal); needs a GPU.
"""
import numpy as np
import pytest

from pcom_b200 import _lib as L
from pcom_b200.model import Batch, Model
from pcom_b200.synth import make_case
from parity_util import STATE_FIELDS, compare
from test_gpu_mixed import BOUNDS, errors

pytestmark = pytest.mark.gpu

# land: none; one that ends inside tiles and crosses the periodic boundary;
# all but a corner
SIZES = [(10, 8, 3), (24, 14, 3), (37, 23, 4), (128, 66, 3), (211, 97, 3)]


def _case(ni, nj, nk, land):
    c = make_case("basin", noise=0.01, glo_ni=ni, glo_nj=nj, nk=nk)
    itn = np.array(c["itn"])
    if land == "band":
        itn[:, : ni // 3] = 0
        itn[:, ni - ni // 8:] = 0
    elif land == "corner":
        itn[nj // 4:] = 0
        itn[:, ni // 4:] = 0
    return dict(c, itn=itn, dtbt=20, dtbc=200)


@pytest.mark.parametrize("land", ["none", "band", "corner"])
@pytest.mark.parametrize("size", SIZES, ids=lambda s: "x".join(map(str, s)))
def test_forms_agree_bit_for_bit(size, land):
    c = _case(*size, land)
    got = {}
    for form in (3, 2, 1):
        m = Model(c)
        L.check(m.lib.pcom_gpu_set_trop_kernel(m.handle, form), "set_trop_kernel")
        m.run(4)
        got[form] = {f: m.field(f) for f in STATE_FIELDS}
        moves = bool((m.static()["lev_u"] >= 1).any())
        m.close()
    # (a sea of one column has no velocity point)
    assert np.isfinite(got[3]["ubc"]).all() and (np.abs(got[3]["ubc"]).max() > 0) == moves
    for form in (2, 1):
        for f in STATE_FIELDS:
            r = compare(got[form][f], got[3][f])
            assert r["unequal"] == 0, f"form {form}, {f}: {r['unequal']} values differ"


@pytest.mark.parametrize("sizes", [[(10, 8), (13, 9), (37, 23)], [(211, 97), (12, 90), (150, 9)], [(128, 66)] * 5],
                         ids=["small", "long", "several launches"])
def test_batch_of_fitted_tiles(sizes):
    """A batch gives each member tiles of its own shape, packed into launches."""
    cases = [_case(ni, nj, 3, "band") for ni, nj in sizes]
    ms = [Model(c) for c in cases]
    b = Batch(ms)
    b.run(4)
    for c, m in zip(cases, ms):
        r = Model(c)
        L.check(r.lib.pcom_gpu_set_trop_kernel(r.handle, 3), "set_trop_kernel")
        r.run(4)
        for f in STATE_FIELDS:
            d = compare(m.field(f), r.field(f))
            assert d["unequal"] == 0, f"{c['itn'].shape}, {f}: {d['unequal']} values differ"
        r.close()
    b.close()
    for m in ms:
        m.close()


@pytest.mark.parametrize("land", ["none", "band"])
@pytest.mark.parametrize("size", [(24, 14, 3), (150, 100, 3), (211, 97, 3)], ids=lambda s: "x".join(map(str, s)))
def test_mixed_resident_shapes(size, land):
    """The mixed resident kernel at a compiled shape and at shapes of the
    domain's own does the multi-tile mixed kernel's arithmetic in code compiled
    apart: half the mixed bounds, as on the 1-degree domain."""
    c = dict(_case(*size, land), dtbt=60, dtbc=3600)
    ms = [Model(c, flags=L.PCOM_PREC_MIXED) for _ in range(2)]
    L.check(ms[1].lib.pcom_gpu_set_trop_kernel(ms[1].handle, 2), "set_trop_kernel")
    for m in ms:
        m.run(6)
    for f, e in errors(ms[0], ms[1]).items():
        assert e <= 0.5 * BOUNDS[f], f"{f} rel RMS {e:.3e}"
    for m in ms:
        m.close()
