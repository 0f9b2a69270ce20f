"""The property update's fields in the place of its inputs, and its two ways to evaluate the fits, over all temperatures."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _setup(name, n, seed):
    import torch
    from laminarsmoke_b200 import lsg, mech
    from tests.test_properties import _cells
    data, species = mech.load(name)
    Y, T, p = _cells(data, species, n, seed)
    dev = lambda x: torch.tensor(np.ascontiguousarray(x), device="cuda")
    return data, lsg.ReactionStep(lsg.Mechanism(data)), Y, T, p, dev


@pytest.mark.parametrize("name", ["h2co", "ch4"])
def test_fields_in_the_place_of_inputs(cuda, name):
    """X over Y, cTot over p and lambda over T: a cell's inputs are read before its fields are written, also where the
    temperature is far outside the fits or not a number."""
    import torch
    from laminarsmoke_b200 import lsg
    n = 200
    _, ctx, Y, T, p, dev = _setup(name, n, 31)
    T[7], T[100], T[150] = 1e-60, np.nan, 1e200
    nc = Y.shape[1]
    want = {k: v.cpu().numpy() for k, v in ctx.properties_device(dev(Y.T), dev(T), dev(p)).items()}
    Yd, Td, pd = dev(Y.T), dev(T), dev(p)
    Dmix = torch.empty_like(Yd)
    fields = lsg.PropertyFields(X=Yd.data_ptr(), cTot=pd.data_ptr(), Dmix=Dmix.data_ptr(), **{"lambda": Td.data_ptr()})
    opt = lsg.PropertyOptions(1, 0, None)
    rc = lsg.lib().lsg_properties_device(ctx.h, n, nc, Yd.data_ptr(), Td.data_ptr(), n, pd.data_ptr(), 0.0, C.byref(opt),
                                         C.byref(fields), n, torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    for k, v in (("X", Yd), ("cTot", pd), ("lambda", Td), ("Dmix", Dmix)):
        np.testing.assert_array_equal(v.cpu().numpy(), want[k], err_msg=k)


@pytest.mark.parametrize("name", ["h2co", "ch4", "syn120t"])
def test_fits_over_all_temperatures(cuda, name):
    """Either way against the oracle from 1e-30 to 1e30 K, where the fits' exponents run through the polynomial
    exponential's range and out of it.  The terms of a fit of magnitude s in sum carry a rounding of some 8 eps s into
    the exponent, hence into the field, beside the 1e-12 of ordinary temperatures."""
    from oracle.properties import OracleProperties
    n = 600
    data, ctx, Y, T, p, dev = _setup(name, n, 37)
    T = np.concatenate([np.logspace(-30, 30, n // 2), np.logspace(0, 5, n - n // 2)])
    got = {k: v.cpu().numpy() for k, v in ctx.properties_device(dev(Y.T), dev(T), dev(p)).items()}
    o = OracleProperties(data)
    with np.errstate(all="ignore"):
        ref = o.evaluate(Y, T, p)
    powers = np.abs(np.log(T))[None, :] ** np.arange(4)[:, None]
    s = {"mu": np.abs(o.eta) @ powers, "lambda": np.abs(o.lam) @ powers, "Dmix": np.abs(o.gam) @ powers}
    for f, size in s.items():
        a, r = got[f], ref[f].T if ref[f].ndim == 2 else ref[f]
        tol = 1e-12 + 8 * 2.220446049250313e-16 * size.max(axis=0)
        fine = np.isfinite(r) & (np.abs(r) > 1e-290) & (np.abs(r) < 1e290) & (tol < 1e-3) & np.isfinite(a)
        assert fine[..., n // 2:].mean() > 0.2
        err = np.abs(a - r) / np.abs(r)
        assert np.all(err[fine] <= np.broadcast_to(tol, err.shape)[fine]), (f, float((err / tol)[fine].max()))
