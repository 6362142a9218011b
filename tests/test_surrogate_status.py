"""What a failed training step raises (host logic, no GPU): ValueError where the
library rejects the arguments, RuntimeError with the status where it fails
otherwise; the step count then stays where it was."""

from __future__ import annotations

import types

import pytest


@pytest.mark.parametrize("status,error,text", [(1, ValueError, "multiple of 128"), (3, RuntimeError, "status 3")])
def test_train_step_raises_by_status(pkg, monkeypatch, status, error, text):
    import torch
    from wrf_jax_b200 import _capi, surrogate as S
    t = torch.zeros(1)
    model = object.__new__(S.SurrogateModel)
    model.step = 7
    for name in ("w", "mw", "vw", "b", "mb", "vb", "wb", "wbt"):
        setattr(model, name, [t] * 4)
    buf = {k: t for k in ("Xb", "Xbt", "Tb", "Y", "dY", "dYt", "part", "loss")}
    buf.update({k: [t] * 3 for k in ("Z", "H", "Ht", "dZ", "dZt")}, gw=[t] * 4, gb=[t] * 4)
    monkeypatch.setattr(model, "_buffers", lambda batch: buf, raising=False)
    monkeypatch.setattr(S, "_stream", lambda stream=None: None)
    monkeypatch.setattr(_capi, "load", lambda: types.SimpleNamespace(rrtmg_sur_train_step=lambda args, s: status))
    with pytest.raises(error, match=text) as raised:
        model.train_step(t, t, torch.zeros(128, dtype=torch.int32), t, lr=1.0e-3)
    assert raised.type is error and model.step == 7
