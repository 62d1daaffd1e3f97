"""What the engine looks at before it hands the tensors of a record to kernels as raw pointers: the device, the rows and the columns that
are read.  The checks are host code, so they are tested here with the host as the engine's device; the engine's own refusals are
tested on a GPU in test_gpu_record_checks.py."""
from __future__ import annotations

import pytest
import torch

from taac_2026_b200 import _lib

CPU = torch.device("cpu")
META = torch.device("meta")      # stands for another device


@pytest.fixture(scope="module")
def native():
    try:
        return _lib.native()
    except (RuntimeError, FileNotFoundError, OSError) as err:
        pytest.skip(f"the host module is not built: {err}")


def _sequence(batch=4, features=2, length=6):
    return dict(values=torch.zeros(batch, features, length, dtype=torch.int64), lengths=torch.zeros(batch, dtype=torch.int64),
                stamps=torch.zeros(batch, length, dtype=torch.int64), request=torch.zeros(batch, dtype=torch.int64))


def _check_sequence(native, t, device=CPU):
    native.check_sequence(device, 4, 2, 6, t["values"], t["lengths"], t["stamps"], t["request"])


def test_a_whole_record_passes(native):
    t = _sequence()
    _check_sequence(native, t)
    _check_sequence(native, {**t, "lengths": None, "stamps": None})


@pytest.mark.parametrize("name", ["values", "lengths", "stamps", "request"])
def test_sequence_tensors_elsewhere_or_of_another_size_are_refused(native, name):
    t = _sequence()
    with pytest.raises(RuntimeError, match="live on"):
        _check_sequence(native, {**t, name: t[name].to(META)})
    with pytest.raises(RuntimeError, match="live on"):
        _check_sequence(native, t, META)
    with pytest.raises(RuntimeError, match="shape"):
        _check_sequence(native, {**t, name: t[name][:3]})           # fewer rows
    with pytest.raises(RuntimeError, match="shape"):
        _check_sequence(native, {**t, name: t[name][None]})
    if t[name].ndim > 1:
        with pytest.raises(RuntimeError, match="shape"):
            _check_sequence(native, {**t, name: t[name][..., :5]})


def _entity(batch=4):
    return dict(ids=torch.zeros(batch, 5, dtype=torch.int64), missing=torch.zeros(batch, 5, dtype=torch.bool), values=torch.zeros(batch, 3),
                values_missing=torch.zeros(batch, 4, dtype=torch.bool))


def _check_entity(native, t, columns=5, fields=4, dense=3):
    native.check_entity(CPU, 4, t["ids"], columns, t["missing"], fields, t["values"], t["values_missing"], dense)


def test_entities(native):
    t = _entity()
    _check_entity(native, t)
    _check_entity(native, {**t, "values_missing": None})
    _check_entity(native, {**t, "missing": None}, fields=0)          # what is not read may be anything
    _check_entity(native, {**t, "values": None, "values_missing": None}, dense=0)
    for name in t:
        with pytest.raises(RuntimeError, match="live on"):
            _check_entity(native, {**t, name: t[name].to(META)})
        with pytest.raises(RuntimeError, match="shape"):
            _check_entity(native, {**t, name: t[name][:2]})
        with pytest.raises(RuntimeError, match="shape"):
            _check_entity(native, {**t, name: torch.cat([t[name], t[name]])})
    for name in ("missing", "values"):
        with pytest.raises(RuntimeError, match="missing"):
            _check_entity(native, {**t, name: None})
    for more in (dict(columns=6), dict(fields=6), dict(dense=5)):
        with pytest.raises(RuntimeError, match="columns|shape"):
            _check_entity(native, t, **more)
