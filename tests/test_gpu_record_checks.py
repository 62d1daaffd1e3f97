"""Malformed records are refused on the host before anything is launched: tensors left on the host, entities and sequences of different
batch sizes, too few columns.  A good record scores as before afterwards."""
from __future__ import annotations

import dataclasses

import pytest
import torch

from conftest import gpu_ready
from taac_2026_b200.onetrans import OneTransInference, random_state_dict
from test_gpu_weight_changes import _batch, _spec

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _need_gpu():
    if not gpu_ready():
        pytest.fail("gpu tests need an sm_100 device and a built libtb200.so")


def _with(batch, part, **changes):
    if part == "seq":
        seq = dataclasses.replace(batch.sequences["seq_a"], **changes)
        return dataclasses.replace(batch, sequences={"seq_a": seq})
    if part == "request":
        return dataclasses.replace(batch, **changes)
    return dataclasses.replace(batch, **{part: dataclasses.replace(getattr(batch, part), **changes)})


def test_malformed_records_are_refused():
    spec, batch = _spec(256), _batch()
    model = OneTransInference(random_state_dict(spec, seed=1, device="cuda", dtype=torch.bfloat16), spec, dtype=torch.bfloat16)
    want = model.scores(batch).clone()
    assert model._executor().assembles_ns_tokens()
    seq = batch.sequences["seq_a"]
    bad = []
    for part, holder, names in (("user", batch.user, ("int_values", "int_missing_mask", "dense_values", "dense_missing_mask")),
                                ("item", batch.item, ("int_values", "int_missing_mask")), ("seq", seq, ("values", "lengths", "timestamps")),
                                ("request", batch, ("request_timestamp",))):
        for name in names:
            t = getattr(holder, name)
            bad += [_with(batch, part, **{name: t.cpu()}), _with(batch, part, **{name: t[:-1]})]
    bad += [_with(batch, "user", int_values=batch.user.int_values[:, :3]), _with(batch, "seq", timestamps=seq.timestamps[:, :-1])]
    for record in bad:
        with pytest.raises(RuntimeError):
            model.scores(record)
    # a prepared result of another batch of the same size cannot serve a record with other positions
    prepared = model.prepare(batch)
    with pytest.raises(RuntimeError, match="shape"):
        model.scores(_with(batch, "seq", values=seq.values[:, :, :-1].contiguous(), timestamps=seq.timestamps[:, :-1].contiguous()), prepared=prepared)
    assert torch.equal(model.scores(batch), want)


def test_another_number_of_blocks_is_refused():
    """The row plan is made for the model's blocks: its totals end where they end."""
    spec, batch = _spec(256), _batch()
    model = OneTransInference(random_state_dict(spec, seed=1, device="cuda", dtype=torch.bfloat16), spec, dtype=torch.bfloat16)
    want = model.scores(batch).clone()
    blocks = model.blocks
    for other in (blocks[:1], blocks + blocks):
        model.blocks = other
        with pytest.raises(RuntimeError, match="blocks"):
            model.scores(batch)
    model.blocks = blocks
    assert torch.equal(model.scores(batch), want)
