"""The Hankel-row kernel in batches: sets, binary masks, fused extremes, groups
side by side and bounded waits. Plans and single matches run the window kernel
where it applies, so these run the same work with the tensor-core path forced
to the Hankel-row kernel, and the shapes that reach it by themselves (templates
of 129 to 256 columns, large binary masks). Bit for bit against the oracle.
"""

import numpy as np
import pytest
import test_gpu_batch as batches
import test_gpu_timeout as timeouts

from imageproc_b200 import _lib
from imageproc_b200 import template_matching as tm
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["0", None], ids=["untuned", "tuned"])
def forced(request, monkeypatch):
    # untuned: sets of up to four unmasked pairs and two masked ones
    monkeypatch.setenv("IPB_TUNING_FILE", "")
    if request.param:
        monkeypatch.setenv("IPB_AUTOTUNE", request.param)
    else:
        monkeypatch.delenv("IPB_AUTOTUNE", raising=False)
    _lib.lib().ipb_batch_tuning_reset()
    tm.set_path(tm.Path.TensorCores)
    yield
    tm.set_path(tm.Path.Auto)
    _lib.lib().ipb_batch_tuning_reset()


@pytest.mark.parametrize("precision", [0, 1])
def test_sets(forced, precision):
    batches.test_pairs_sharing_images_form_sets_bit_exact(precision)


def test_mixed_pairs_with_fused_extremes(forced):
    batches.test_batch_mixed_pairs_bit_exact_with_fused_extremes(3)


def test_plan_replay(forced):
    batches.test_batch_plan_graph_replay()


def test_groups_side_by_side(forced):
    batches.test_batch_groups_side_by_side_claim_every_tile_once()


def test_more_problems_than_fit_in_kernel_parameters(forced):
    batches.test_batch_of_more_problems_than_fit_in_kernel_parameters()


def test_shapes_that_the_window_kernel_leaves(monkeypatch):
    # by themselves, no path forced: wide templates, large binary masks, and a
    # masked pair the window kernel could take in a group with one it cannot
    import torch

    from imageproc_b200 import device
    monkeypatch.setenv("IPB_TUNING_FILE", "")
    _lib.lib().ipb_batch_tuning_reset()
    tm.set_path(tm.Path.Auto)
    g = np.random.default_rng(29)
    image = g.integers(0, 256, (300, 517), dtype=np.uint8)
    items = []
    for h, w, masked in ((40, 129, False), (100, 256, False), (128, 128, True), (96, 82, True), (30, 70, True)):
        template = g.integers(0, 256, (h, w), dtype=np.uint8)
        mask = (g.random((h, w)) < 0.8).astype(np.uint8) if masked else None
        items += [(image, template, method, mask) for method in range(4)]
    batch = device.Batch(batches._to_device_shared(items))
    plan = device.BatchPlan(batch)
    assert plan.info()["tensor_pairs"] == len(items)
    for _ in range(2):
        for out in batch.outs:
            out.fill_(-1.0)
        plan.launch()
        torch.cuda.synchronize()
        batches._check(items, batch.outs, batch.extremes_host())
    plan.close()
    for image, template, method, mask in items:
        got = tm.match_template(image, template, method) if mask is None else \
            tm.match_template_with_mask(image, template, method, mask)
        assert np.array_equal(batches.bits(got),
                              batches.bits(O.match_exact(image, template, method, mask, precision=0)))


@pytest.fixture
def tiny_budget():
    L = _lib.lib()
    yield L
    timeouts._stall(L, False)
    tm.set_path(tm.Path.Auto)


def test_wait_runs_out_then_context_recovers(tiny_budget, monkeypatch):
    # the single-template timeout test asks for Path.Auto: here it is given the
    # Hankel-row kernel instead
    set_path = tm.set_path
    monkeypatch.setattr(tm, "set_path", lambda p: set_path(tm.Path.TensorCores if p == tm.Path.Auto else p))
    timeouts.test_single_template_wait_runs_out_then_context_recovers(tiny_budget)
    assert tm.get_path() == tm.Path.TensorCores
    monkeypatch.undo()
