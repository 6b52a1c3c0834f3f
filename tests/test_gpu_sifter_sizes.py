"""The sifter's kernels at the edges of their tiles (32-candidate tiles split over clusters, 16-candidate blocks,
32-candidate pipeline steps), against the numpy oracle with the kernels' bf16 rounding points, and with patches that
do not start on a 16-byte boundary. One rounding of an activation to bf16 is 2^-9 of it; over the 256 and 128 terms of
the next layers a few flipped roundings stay below 5e-3 of the result's norm."""

import numpy as np
import pytest

import sifter_oracle as SO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 33, 65, 300, 1024])
def test_sifter_batch_sizes(pb2lib, n):
    import torch
    from pirate_b200.sifter import PATCH_LEN, Sifter
    rng = np.random.default_rng(n)
    s = Sifter(device=0, max_batch=1024, seed=2)
    p = s.get_params()
    p += 0.01 * rng.standard_normal(p.size).astype(np.float32)
    s.set_params(p)
    x = rng.standard_normal((n, PATCH_LEN)).astype(np.float16)
    y = (rng.random(n) < 0.5).astype(np.float32)
    buf = torch.zeros(n * PATCH_LEN + 8, dtype=torch.float16, device="cuda")
    got = []
    for off in (0, 1):   # 16-byte aligned, and not
        xd = buf[off:off + n * PATCH_LEN].view(n, PATCH_LEN)
        xd.copy_(torch.from_numpy(x))
        loss, g = s.gradients(xd, torch.from_numpy(y).cuda())
        got.append((s.forward(xd).cpu().numpy(), loss, g))
    z, c = SO.forward(p, x)
    wl, wg = SO.gradients(p, x, y)
    for zg, loss, g in got:
        assert np.linalg.norm(zg - z) <= 5e-3 * np.linalg.norm(z) + 1e-3
        assert abs(loss - wl) <= 5e-3 * abs(wl) + 1e-4
        for a, b in zip(SO.split(g), SO.split(wg)):
            assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b) + 1e-7
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][2], got[1][2])


def test_sifter_train_step_is_adam_on_gradients(pb2lib):
    import torch
    from pirate_b200.sifter import PATCH_LEN, Sifter
    rng = np.random.default_rng(0)
    s = Sifter(device=0, max_batch=64, seed=3)
    p = s.get_params().astype(np.float64)
    m, v = np.zeros_like(p), np.zeros_like(p)
    for k in range(1, 4):
        x = torch.from_numpy(rng.standard_normal((50, PATCH_LEN)).astype(np.float16)).cuda()
        y = torch.from_numpy((rng.random(50) < 0.5).astype(np.float32)).cuda()
        loss, g = s.gradients(x, y)
        assert s.train_step(x, y, 1e-3) == loss
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g.astype(np.float64) ** 2
        p = p - 1e-3 * (m / (1 - 0.9 ** k)) / (np.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
        # fp32 moments and update: a few ulp of parameters below 1, and of a step of about 1e-3
        assert np.abs(s.get_params() - p).max() <= 2e-6
