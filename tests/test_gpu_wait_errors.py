"""A bounded wait that ran out inside a kernel (its word in page-locked memory set, here by the host) is
reported by whatever next hands results to the host, once."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture()
def ctx():
    import tenetgb

    return tenetgb.Context(0)


def _word(ctx):
    f = getattr(ctx.lib, "_Z15wait_error_wordP6tn_ctxPPi")  # tn_status_t wait_error_word(tn_ctx*, int**)
    f.argtypes, f.restype = [C.c_void_p, C.POINTER(C.POINTER(C.c_int))], C.c_int
    p = C.POINTER(C.c_int)()
    assert f(ctx.h, C.byref(p)) == 0
    return p


def _mps(ctx):
    import tenetgb

    rng = np.random.default_rng(1)
    bonds = [1, 2, 4, 2, 1]
    sites = [rng.standard_normal((a, 2, b)) + 1j * rng.standard_normal((a, 2, b)) for a, b in zip(bonds, bonds[1:])]
    return tenetgb.MPS(sites, ctx=ctx)


def _read_backs(ctx, tmp_path):
    import tenetgb
    from tenetgb.group import MPSGroup

    psi = _mps(ctx)
    bond = _mps(ctx)
    bond.canonize_(tenetgb.BondCanonical(2, 3))
    random_group = lambda: MPSGroup.random([5, 6], [4, 3], ctx=ctx)
    group = random_group()
    t = tenetgb.DeviceTensor.from_numpy(ctx, np.ones((4, 4), complex))
    return {
        "sync": ctx.sync,
        "tensor": t.numpy,
        "sites": psi.sites,
        "site": lambda: psi.site(2),
        "norm": psi.norm,
        "lambda": bond.lambda_,
        "save": lambda: psi.save(str(tmp_path / "psi")),
        "save_lambda": lambda: bond.save(str(tmp_path / "bond")),
        "group_sites": lambda: group.sites(1),
        "group_norms": lambda: random_group().canonize_compress_norm(2),
    }


@pytest.mark.parametrize("name", ["sync", "tensor", "sites", "site", "norm", "lambda", "save", "save_lambda", "group_sites",
                                  "group_norms"])
def test_reported_once(ctx, tmp_path, name):
    from tenetgb import _lib

    call = _read_backs(ctx, tmp_path)[name]
    call()
    _word(ctx)[0] = 1
    with pytest.raises(_lib.DeviceTimeoutError):
        call()
    call()

