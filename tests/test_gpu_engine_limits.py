"""Batches and widths at the far end of what the engine takes."""
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


def test_more_samples_than_a_grid_dimension():
    """65 537 samples of at most four events: no sequence row survives the first block, which then runs for the last rows alone.  Rows are
    independent and no product splits its sum by the number of rows at these sizes, so smaller batches give the same bits."""
    spec = _spec(256)
    model = OneTransInference(random_state_dict(spec, seed=1, device="cuda", dtype=torch.bfloat16), spec, dtype=torch.bfloat16)
    batch = _batch(65_537)
    seq = batch.sequences["seq_a"]
    lens = seq.lengths.clamp_max(4)
    values = torch.where(torch.arange(seq.values.shape[2], device="cuda") < lens[:, None, None], seq.values, 0)
    batch = dataclasses.replace(batch, sequences={"seq_a": dataclasses.replace(seq, values=values, lengths=lens)})
    assert torch.equal(model.scores(batch), model.scores(batch, micro_batch=20_000))


@pytest.mark.parametrize("dense", [0, 4])
def test_wide_model_without_dense_features(dense):
    """d_model 1536: the statistics token does not fit the small-token kernel, whether or not there are dense ones.  The padded layout
    computes the same scores with other kernels: bf16 results around one half, a few units of 2^-9 of the logits apart."""
    spec = dataclasses.replace(_spec(1536, heads=24, dense=dense), num_blocks=1, user_ns_tokens=1, item_ns_tokens=1)
    weights = random_state_dict(spec, seed=2, device="cuda", dtype=torch.bfloat16)
    batch = _batch(9, dense=dense)
    got = OneTransInference(weights, spec, dtype=torch.bfloat16).scores(batch)
    want = OneTransInference(weights, spec, dtype=torch.bfloat16, packed=False).scores(batch)
    torch.testing.assert_close(got, want, rtol=0, atol=4e-3)
