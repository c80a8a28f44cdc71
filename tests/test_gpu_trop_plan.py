"""The barotropic kernel's form is chosen, and its memory taken, when the
static data are uploaded: a new model's first step allocates nothing, and a
large domain for whose packed coefficients no memory is left still runs, in
the generic form, with the same results; needs a GPU."""
import ctypes as C

import numpy as np
import pytest

from pcom_b200 import _lib as L
from pcom_b200.model import Model
from pcom_b200.synth import make_case
from parity_util import STATE_FIELDS, compare

pytestmark = pytest.mark.gpu

BIG = (720, 320, 3)  # the half-degree globe: more tiles than SMs at any resident shape


def _case():
    return dict(make_case("global05", noise=0.01, nk=BIG[2]), dtbt=20, dtbc=200)


@pytest.mark.parametrize("flags", [L.PCOM_PREC_FP64, L.PCOM_PREC_MIXED], ids=["fp64", "mixed"])
def test_first_step_allocates_nothing(flags):
    import torch

    c = _case()
    for trial in range(2):  # the first model's step loads the kernels
        m = Model(c, flags=flags)
        free = torch.cuda.mem_get_info()[0]
        m.run(1)
        taken = free - torch.cuda.mem_get_info()[0]
        m.close()
    assert taken == 0, f"the first step took {taken} bytes"


def test_no_memory_for_packed_coefficients():
    import torch

    ref = Model(_case())
    lib = ref.lib
    st, static = {f: ref.field(f) for f in ("tc", "sc")}, L.Static()
    L.check(lib.pcom_model_static(ref._m, C.byref(static)), "static")
    d = L.Dims(ref.glo_ni, ref.glo_nj, ref.nk, ref.ni, ref.nj, ref.case["dtbt"], ref.case["dtbc"], 0, 0)
    h = C.c_void_p()
    L.check(lib.pcom_gpu_create(C.byref(d), C.byref(h)), "create")
    # 16 MiB stay free; the coefficients are 20 values for each of 724 x 322 points (35 MiB)
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - (16 << 20), dtype=torch.uint8, device="cuda")
    try:
        rc = lib.pcom_gpu_upload_static(h, C.byref(static))
    finally:
        del held
        torch.cuda.empty_cache()
    L.check(rc, "upload_static")
    state = L.State()
    state.tc, state.sc = (np.ascontiguousarray(st[f]).ctypes.data_as(L.dbl_p) for f in ("tc", "sc"))
    L.check(lib.pcom_gpu_set_state(h, C.byref(state)), "set_state")
    forcing = ref.int_bnd()
    frc = L.Forcing(*[forcing[k].ctypes.data_as(L.dbl_p) for k in ("taux", "tauy", "t", "s", "pa", "fw")])
    L.check(lib.pcom_gpu_set_forcing(h, C.byref(frc)), "set_forcing")
    L.check(lib.pcom_gpu_den_prho(h), "den_prho")
    launches = []
    for it in (1, 2, 3):
        before = lib.pcom_gpu_launch_count(h)
        L.check(lib.pcom_gpu_step(h, it), "step")
        launches.append(lib.pcom_gpu_launch_count(h) - before)
    ref.run(1)
    before = ref.launch_count()
    ref.run(1)
    # (the form with packed coefficients launches their packing as well)
    assert launches[1] == ref.launch_count() - before - 1
    ref.run(1)
    assert ref.glo_ni == BIG[0] and np.isfinite(ref.field("ubc")).all()
    for f in STATE_FIELDS:
        a = np.zeros(int(lib.pcom_gpu_field_size(h, f.encode())))
        L.check(lib.pcom_gpu_get_field(h, f.encode(), a.ctypes.data_as(L.dbl_p), a.size), f)
        b = ref.field(f)
        r = compare(a.reshape(b.shape), b)
        assert r["unequal"] == 0, f"{f}: {r['unequal']} values differ"
    lib.pcom_gpu_destroy(h)
    ref.close()
