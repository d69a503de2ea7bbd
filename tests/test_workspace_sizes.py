"""Workspace sizes never fall when the call grows: a workspace made for the largest population serves every
smaller one, and a buffer whose address a captured graph holds is never replaced by a smaller call."""
import pytest

from altar_gb300 import _native

# around every launch rule (multiples of 16 to 9,728 chains and their neighbours), coarsely to 10^6
SIZES = sorted({max(1, q * k + d) for k in (16, 128, 256, 1024, 2432, 9728) for q in range(20) for d in (-1, 0, 1)}
               | set(range(2700, 3400, 7)) | {3071, 3072, 3073} | set(range(5000, 1000001, 19937)))


def _never_falls(f):
    last = 0
    for n in SIZES:
        need = f(n)
        assert need >= last > -1, f"{n} chains need {need} bytes, fewer chains {last}"
        last = need


@pytest.mark.parametrize("model", [_native.AG_MODEL_CDM, _native.AG_MODEL_MOGI])
def test_forward(native_lib, model):
    _never_falls(lambda n: native_lib.ag_forward_workspace_bytes(model, n))


@pytest.mark.parametrize("p", [1, 4, 10, 21, 22, 100, 512])
def test_covariance(native_lib, p):
    _never_falls(lambda n: native_lib.ag_sigma_workspace_bytes(n, p))


def test_stage(native_lib):
    _never_falls(native_lib.ag_cov_workspace_bytes)
    _never_falls(native_lib.ag_resample_workspace_bytes)


@pytest.mark.parametrize("m", [1, 300, 4950])
def test_products(native_lib, m):
    _never_falls(lambda n: native_lib.ag_linear_workspace_bytes(m, 61, n))
    _never_falls(lambda n: native_lib.ag_whiten_workspace_bytes(m, n))
