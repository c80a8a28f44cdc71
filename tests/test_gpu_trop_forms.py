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


def _globe(ni, nj, nk, land):
    """The same land on a periodic 80S-80N grid without walls in x."""
    c = _case(ni, nj, nk, "none")
    itn = np.full((nj, ni), nk, np.int32)
    itn[[0, -1]] = 0
    if land == "band":
        itn[:, ni // 8: ni // 8 + ni // 2] = 0
        itn[nj // 2: nj // 2 + nj // 8] = 0
    return dict(c, itn=itn, lat=np.linspace(-80.0, 80.0, nj), lon=(np.arange(ni) + 0.5) * (360.0 / ni))


def _tiles(m, tx, ty):
    """Tiles of a domain (rows of tx columns) that have sea, and those that have none."""
    st = m.static()
    sea = ((st["lev_t"] >= 1) | (st["lev_u"] >= 1))[:, 1:-1]
    nj, ni = sea.shape
    wet = [(j, i) for j in range(0, nj, ty) for i in range(0, ni, tx) if sea[j:j + ty, i:i + tx].any()]
    dry = [(j, i) for j in range(0, nj, ty) for i in range(0, ni, tx) if not sea[j:j + ty, i:i + tx].any()]
    return wet, dry


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("size,land", [((720, 320, 3), "none"), ((720, 320, 3), "band"), ((611, 253, 3), "band"),
                                       ((467, 217, 2), "none")], ids=lambda v: v if isinstance(v, str) else "x".join(map(str, v)))
def test_several_tiles_per_cta(size, land):
    """Domains with more tiles with sea than SMs: the next tile's loads behind
    the current one's stages, the walk forwards and backwards, the two sets of
    metric vectors, an uneven number of tiles per CTA, and tiles without sea
    beside all that."""
    c = _globe(*size, land)
    got = {}
    for form in (3, 2):
        m = Model(c)
        L.check(m.lib.pcom_gpu_set_trop_kernel(m.handle, form), "set_trop_kernel")
        m.run(3)
        got[form] = {f: m.field(f) for f in STATE_FIELDS}
        counts = [tuple(map(len, _tiles(m, *shape))) for shape in ((24, 14), (20, 16), (28, 12))]
        m.close()
    for wet, dry in counts:
        assert wet > _sms() and wet % _sms() and (land == "none" or dry > 0), counts
    assert np.isfinite(got[3]["ubc"]).all() and np.abs(got[3]["ubc"]).max() > 0
    for f in STATE_FIELDS:
        r = compare(got[2][f], got[3][f])
        assert r["unequal"] == 0, f"{f}: {r['unequal']} values differ"


def test_mixed_dry_tiles_are_skipped():
    """A mixed domain where leaving out the tiles without sea saves a CTA a
    tile per substep, against the same domain with a one-point lake in every
    such tile, where all are walked.  (T and S are level means in 1/16ths, so
    the lakes leave the reference profile as it is.)  The points of those
    tiles hold the same sums; the sea, in code compiled apart, agrees to half
    the mixed bounds."""
    ni, nj, nk = 720, 320, 3
    c = _globe(ni, nj, nk, "band")
    pt = np.empty((nk, nj, ni))
    pt[:] = (np.round(np.asarray(c["tmn"]) * 16) / 16)[:, None, None]
    c = dict(c, pt=pt, sa=np.full((nk, nj, ni), 35.0))
    ms = [Model(c, flags=L.PCOM_PREC_MIXED)]
    wet, dry = _tiles(ms[0], 32, 10)
    for per_sm in (1, 2, 3, 4):  # 512 threads per CTA
        n = per_sm * _sms()
        assert len(wet) + len(dry) > n and -(-len(wet) // n) < -(-(len(wet) + len(dry)) // n)
    itn = c["itn"].copy()
    land = np.zeros((nj + 2, ni + 2), bool)  # the dry tiles' points, without the lakes
    for j, i in dry:
        land[j:j + 10, i + 1:min(i + 33, ni + 1)] = True
        lj, li = min(j + 5, nj), min(i + 16, ni - 1)
        if 1 <= lj - 1 < nj - 1:
            itn[lj - 1, li] = 1
            land[lj, li + 1] = False
    ms.append(Model(dict(c, itn=itn), flags=L.PCOM_PREC_MIXED))
    left = _tiles(ms[1], 32, 10)[1]
    assert len(wet) + len(dry) - len(left) > 4 * _sms() and land.sum() > 10000
    for m in ms:
        m.run(4)
    for f, e in errors(ms[1], ms[0]).items():
        assert e <= 0.5 * BOUNDS[f], f"{f} rel RMS {e:.3e}"
    assert np.abs(ms[0].field("ubc")).max() > 0
    for f in ("ubc", "vbc", "ubp", "vbp", "chc", "chp", "mch", "mch2", "acch"):
        r = compare(ms[0].field(f), ms[1].field(f), land)
        assert r["unequal"] == 0, f"{f}: {r['unequal']} land values differ"
    for m in ms:
        m.close()


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
