"""The window kernel (staged image tiles read in place as an MMA operand)
against the oracle, bit for bit.

Shapes sit at the kernel's edges: template widths where the K of the MMAs or
the staged pitch steps (1, 2, 17, 18, 33, 34, 49, 50, 81, 82, 113, 114, 128),
template heights below, at and above a tile's rows per lane group and at the
limits of the block slots (1, 7, 8, 9, 64, 65, 127, 128), maps of one row, one
column, one position, a tile and one more, and image rows on 16-byte, 4-byte
and odd boundaries.
"""

import numpy as np
import pytest

from imageproc_b200 import template_matching as tm
from oracle import oracle as O

pytestmark = pytest.mark.gpu
M = tm.MatchTemplateMethod

# (image width, height), (template width, height)
SHAPES = [
    ((128, 40), (1, 1)), ((255, 33), (2, 7)), ((144, 23), (17, 8)), ((145, 200), (18, 9)),
    ((161, 97), (33, 65)), ((34, 150), (34, 1)), ((513, 128), (49, 128)), ((178, 177), (50, 50)),
    ((208, 271), (81, 128)), ((700, 65), (82, 64)), ((1300, 300), (113, 33)), ((113, 1000), (113, 127)),
    ((242, 143), (114, 16)), ((256, 255), (128, 128)), ((128, 128), (128, 128)), ((1024, 768), (64, 64)),
    ((2000, 1111), (31, 5)),
]


@pytest.fixture(autouse=True)
def _restore():
    old_p, old_path = tm.get_precision(), tm.get_path()
    tm.set_path(tm.Path.Auto)
    yield
    tm.set_precision(old_p)
    tm.set_path(old_path)


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def scene(W, H, w, h):
    g = np.random.default_rng(W * 7 + H * 5 + w * 3 + h)
    image = g.integers(0, 256, (H, W), dtype=np.uint8)
    image[: H // 3, : W // 2] = 0  # zero norms
    image[H // 2:, W // 2:] = 255
    return image, g.integers(0, 256, (h, w), dtype=np.uint8), (g.random((h, w)) < 0.7).astype(np.uint8)


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0][0]}x{s[0][1]}_t{s[1][0]}x{s[1][1]}")
def test_window_kernel_bit_exact(shape):
    (W, H), (w, h) = shape
    image, template, mask = scene(W, H, w, h)
    for method in M:
        for m in (None, mask):
            got = tm.match_template(image, template, method) if m is None else \
                tm.match_template_with_mask(image, template, method, m)
            exp = O.match_exact(image, template, method, m, precision=0)
            bad = np.argwhere(bits(got) != bits(exp))
            assert bad.size == 0, (method, m is not None, bad[:3])


@pytest.mark.parametrize("offset", [0, 1, 2, 4, 8])
def test_window_kernel_unaligned_buffers_and_sets(offset, tmp_path, monkeypatch):
    # images, templates and masks at odd addresses; sets of one image whose
    # members differ in template, method and need of the window sums, binary
    # masks among them, untuned so that every group runs on the window kernel
    import torch

    from imageproc_b200 import _lib, device
    monkeypatch.setenv("IPB_AUTOTUNE", "0")
    monkeypatch.setenv("IPB_TUNING_FILE", "")
    _lib.lib().ipb_batch_tuning_reset()

    def dev(a):
        buf = torch.zeros(a.size + 64, dtype=torch.uint8, device="cuda")
        view = buf[offset:offset + a.size].view(a.shape)
        view.copy_(torch.from_numpy(a))
        return view

    items, dev_items = [], []
    for W, H, w, h in ((512, 300, 40, 24), (301, 260, 64, 64), (640, 129, 8, 100), (700, 500, 64, 40),
                       (400, 300, 128, 128)):
        image, t0, mask = scene(W, H, w, h)
        t1 = t0[::-1].copy()
        di, d0, d1, dm = dev(image), dev(t0), dev(t1), dev(mask)
        # sets of four: one template three times, then another
        for t, d, method in ((t0, d0, 2), (t0, d0, 3), (t1, d1, 0), (t0, d0, 1)):
            items += [(image, t, method, None), (image, t, method, mask)]
            dev_items += [(di, d, method), (di, d, method, dm)]
    batch = device.Batch(dev_items)
    plan = device.BatchPlan(batch)
    for _ in range(2):
        for o in batch.outs:
            o.fill_(-1.0)
        plan.launch()
        torch.cuda.synchronize()
        for k, ((image, t, method, mask), out, e) in enumerate(zip(items, batch.outs, batch.extremes_host())):
            exp = O.match_exact(image, t, method, mask, precision=0)
            bad = np.argwhere(bits(out.cpu().numpy()) != bits(exp))
            assert bad.size == 0, (k, bad[:3])
            mx, mn, mxl, mnl = O.find_extremes(exp)
            assert (e.max_value, e.min_value, e.max_value_location, e.min_value_location) == \
                (float(mx), float(mn), mxl, mnl), k
    plan.close()


@pytest.mark.parametrize("tune", [False, True])
def test_window_kernel_mixed_group(tune, tmp_path, monkeypatch):
    # more problems in a launch than its parameters hold, of unequal sizes: a
    # CTA passes from templates of one chunk to ones over both block slots and
    # in many chunks, from sets that need window sums to sets that do not, and
    # takes several tiles of one template in a row, staged by tensor copies
    # (rows on 16-byte boundaries) and without
    import torch

    from imageproc_b200 import _lib, device
    monkeypatch.setenv("IPB_AUTOTUNE", "1" if tune else "0")
    monkeypatch.setenv("IPB_TUNING_FILE", "")
    _lib.lib().ipb_batch_tuning_reset()
    sizes = [(2720, 2704, 25, 6, 2), (2720, 1500, 9, 4, 3), (1601, 700, 31, 17, 0), (640, 400, 18, 120, 1),
             (333, 444, 12, 97, 2), (512, 512, 29, 61, 3), (410, 300, 17, 1, 2), (800, 600, 32, 45, 1),
             (257, 258, 8, 109, 0), (1200, 900, 24, 30, 2), (448, 300, 30, 104, 3)]
    items, dev_items = [], []
    for W, H, w, h, method in sizes:
        image, t, _ = scene(W, H, w, h)
        items.append((image, t, method))
        dev_items.append((torch.from_numpy(image).cuda(), torch.from_numpy(t).cuda(), method))
    batch = device.Batch(dev_items)
    plan = device.BatchPlan(batch)
    exp = [O.match_exact(image, t, method, precision=0) for image, t, method in items]
    for _ in range(3):
        for o in batch.outs:
            o.fill_(-1.0)
        plan.launch()
        torch.cuda.synchronize()
        for k, (want, out) in enumerate(zip(exp, batch.outs)):
            bad = np.argwhere(bits(out.cpu().numpy()) != bits(want))
            assert bad.size == 0, (sizes[k], bad[:3])
    plan.close()


@pytest.mark.parametrize("rows", [16, 32, 64, 128])
@pytest.mark.parametrize("members", [1, 4])
def test_window_kernel_short_tiles(rows, members, tmp_path, monkeypatch):
    # tiles of a few MMAs, many per CTA, of one template that stays in its
    # slots: the roles run as far ahead of each other as they can
    import torch

    from imageproc_b200 import _lib, device
    W, H, w, h = 1920, 1080, 8, 8
    image, t0, _ = scene(W, H, w, h)
    pos = (W - w + 1) * (H - h + 1) * members
    f = tmp_path / "tuning.txt"
    f.write_text(f"group2 8 0 8 {pos.bit_length() - 1} 10 {100 + members} 0 {rows} {members}\n")
    monkeypatch.setenv("IPB_TUNING_FILE", str(f))
    _lib.lib().ipb_batch_tuning_reset()
    di, dt = torch.from_numpy(image).cuda(), torch.from_numpy(t0).cuda()
    batch = device.Batch([(di, dt, k) for k in range(members)])
    plan = device.BatchPlan(batch)
    assert plan.info()["launches"][0]["tile_rows"] == rows
    for k in range(20):
        if k == 19:
            for o in batch.outs:
                o.fill_(-1.0)
        plan.launch()
    torch.cuda.synchronize()
    batch.extremes_host()
    for k, out in enumerate(batch.outs):
        bad = np.argwhere(bits(out.cpu().numpy()) != bits(O.match_exact(image, t0, k, precision=0)))
        assert bad.size == 0, (k, bad[:3])
    plan.close()
    _lib.lib().ipb_batch_tuning_reset()


@pytest.mark.parametrize("W,H,w,h,rows", [(1280, 957, 16, 16, 128), (1283, 957, 8, 8, 128), (512, 512, 16, 16, 16),
                                          (4095, 3000, 9, 16, 128)])
def test_estimate_counts_a_tiles_own_cost(W, H, w, h, rows, monkeypatch):
    # measured, 16 to 128 rows per tile: 1280 x 957 27, 22, 20 and 19 us, 1283 x
    # 957 26, 18, 18 and 16, 512 x 512 12, 13, 17 and 20, 4095 x 3000 180, 104,
    # 73 and 60
    import torch

    from imageproc_b200 import _lib, device
    monkeypatch.setenv("IPB_AUTOTUNE", "0")
    monkeypatch.setenv("IPB_TUNING_FILE", "")
    _lib.lib().ipb_batch_tuning_reset()
    image, template, _ = scene(W, H, w, h)
    batch = device.Batch([(torch.from_numpy(image).cuda(), torch.from_numpy(template).cuda(), 0)], extremes=False)
    plan = device.BatchPlan(batch)
    assert [g["tile_rows"] for g in plan.info()["launches"]] == [rows]
    plan.close()


def test_cached_height_without_a_plan_falls_back_to_the_estimate(tmp_path, monkeypatch):
    # 128 rows fit masked templates of up to 113 x 64, and a narrower one of the
    # same key may have left them in the file: a 128 x 64 one takes what it would
    # take without a file
    import torch

    from imageproc_b200 import _lib, device
    W, H, w, h = 1920, 1080, 128, 64  # more tiles than SMs: the estimate makes sets of two
    image, t0, mask = scene(W, H, w, h)
    di, d0, dm = (torch.from_numpy(a).cuda() for a in (image, t0, mask))
    batch = device.Batch([(di, d0, k, dm) for k in (1, 3)])
    monkeypatch.setenv("IPB_AUTOTUNE", "0")
    monkeypatch.setenv("IPB_TUNING_FILE", "")
    _lib.lib().ipb_batch_tuning_reset()
    plan = device.BatchPlan(batch)
    untuned = plan.info()["launches"]
    plan.close()
    pos = 2 * (W - w + 1) * (H - h + 1)
    f = tmp_path / "tuning.txt"
    line = f"group2 32 1 {h} {pos.bit_length() - 1} 10 102 0 128 1\n"
    f.write_text(line)
    monkeypatch.setenv("IPB_TUNING_FILE", str(f))
    monkeypatch.delenv("IPB_AUTOTUNE")
    _lib.lib().ipb_batch_tuning_reset()
    plan = device.BatchPlan(batch)
    assert f.read_text() == line  # the key was found
    assert plan.info()["launches"] == untuned and untuned[0]["set_size"] == 2
    plan.launch()
    torch.cuda.synchronize()
    for k, out in zip((1, 3), batch.outs):
        assert np.array_equal(bits(out.cpu().numpy()), bits(O.match_exact(image, t0, k, mask, precision=0)))
    plan.close()
    _lib.lib().ipb_batch_tuning_reset()
