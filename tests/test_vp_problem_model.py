"""VpProblem forms its model on the device only where that is the model and the
gradient that the host's form gives: reversed or NaN limits (np.clip's results),
limits that are arrays or none, an own `full` and a context with models or
gradients of its own take the host's form."""
import numpy as np
import pytest

NZ, NX = 12, 7
G = [np.full((NZ, NX), v) for v in (2.0, 3.0, 5.0)]


def _context(fw, base):
    class Context(base):
        def __init__(self):
            self.model = None

        def stage_shots(self, *args, **kwargs):
            pass

        def set_illumination(self, on):
            pass

        def set_model(self, *model):
            self.model = model

        def run(self, calc_id):
            pass

        def fetch(self, misfit=True, grads=False, n_shots=0):
            return (1.0, *G, None) if grads else (1.0, None, None, None, None)

    return Context()


def _problem(cls, ctx, **limits):
    rng = np.random.default_rng(0)
    mask = (rng.uniform(size=(NZ, NX)) > 0.3).astype(float)
    return cls(ctx, np.zeros((1, 4)), [0], None, rng.uniform(1500, 3000, (NZ, NX)), np.ones((NZ, NX)), mask, **limits)


@pytest.mark.parametrize("own", ["duck", "subclass"])
def test_own_context(own, fw):
    from fwiflow_gb300 import inversion

    ctx = _context(fw, object if own == "duck" else fw.FwiContext)
    p = _problem(inversion.VpProblem, ctx)
    vp = p.vp0 + 10.0
    J, g, grads, _ = p.misfit_grad(vp)
    for a, b in zip(ctx.model, inversion.moduli_of_vp(p.full(vp))):
        assert np.array_equal(a, b)
    assert np.array_equal(g, inversion.chain_to_vp(p.full(vp), *G) * p.mask)
    assert p.misfit(vp) == 1.0
    ctx._h = None


@pytest.mark.parametrize("limits", [dict(vmin=3000.0, vmax=1500.0), dict(vmin=float("nan")), dict(vmin=None),
                                    dict(vmax=np.full((NZ, NX), 2500.0)), "full"])
def test_own_limits(limits, fw, monkeypatch):
    from fwiflow_gb300 import inversion

    class Own(inversion.VpProblem):
        def full(self, vp):
            return np.maximum(super().full(vp), 2000.0)

    monkeypatch.setattr(fw.FwiContext, "__init__", lambda self: None)
    monkeypatch.setattr(fw.FwiContext, "__del__", lambda self: None, raising=False)
    calls = []
    for name, result in (("stage_shots", None), ("set_illumination", None), ("run", None),
                         ("fetch", (1.0, *G, None))):
        monkeypatch.setattr(fw.FwiContext, name, lambda self, *a, _r=result, **k: _r)
    monkeypatch.setattr(fw.FwiContext, "set_model", lambda self, *m: calls.append(m))
    own = limits == "full"
    p = _problem(Own if own else inversion.VpProblem, fw.FwiContext(), **({} if own else limits))
    vp = p.vp0 + 10.0
    _, g, _, _ = p.misfit_grad(vp)
    for a, b in zip(calls[0], inversion.moduli_of_vp(p.full(vp))):
        assert np.array_equal(a, b, equal_nan=True)
    assert np.array_equal(g, inversion.chain_to_vp(p.full(vp), *G) * p.mask, equal_nan=True)
