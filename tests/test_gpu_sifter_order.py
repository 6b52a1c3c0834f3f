"""The order of the sifter's sums: every product is one chain over its inner index and every bias gradient one chain
over the candidates, for every batch size. So a candidate's score does not depend on the batch that it is scored in,
and scores, loss, gradients and trained parameters are those recorded from the kernels that first computed them (one
GEMM launch per product), bit for bit."""

import zlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Candidates: CRC-32 of the scores, the loss, the gradients, three training losses and the trained parameters.
RECORDED = {
    1: (0x42b25c68, 0x255d69e0, 0x197ff0bb, 0xc4dd5703, 0xc350c865),
    8: (0x27da6fe4, 0x493de933, 0x6f85dd5b, 0x487470f9, 0xa8bf3226),
    17: (0xb5851515, 0xbb8f207d, 0x6ce3703d, 0x48c4bf00, 0x4c08a705),
    33: (0x162fd072, 0xee610d24, 0x904117cb, 0xedde2b93, 0x467a065a),
    64: (0x5b75e21f, 0xdf78afb7, 0xc8e5b954, 0x4e84535b, 0x1346eda7),
    100: (0x9b57877d, 0x35ac6147, 0x9be773ef, 0x7de2dcfa, 0x58a10b13),
    300: (0x7929d22d, 0x60dbe639, 0xf2cfb775, 0xb79922ca, 0xaf5ac636),
    512: (0x1e35c121, 0x6141da95, 0x65e23734, 0x65b134ef, 0xb3919044),
    1000: (0x0ec48e65, 0xd70acc55, 0x5ed1881a, 0x37b59460, 0xb7a1bec4),
    1024: (0x20d36f85, 0x3f79e22d, 0x633ef09e, 0xf97aeb8f, 0x6ba108ce),
}


def _sifter(rng):
    from pirate_b200.sifter import Sifter
    s = Sifter(device=0, max_batch=1024, seed=2)
    p = s.get_params()
    s.set_params(p + 0.01 * rng.standard_normal(p.size).astype(np.float32))
    return s


def _crc(a):
    # + 0: zeros of either sign are the same
    return zlib.crc32(np.ascontiguousarray(a + np.float32(0), dtype=np.float32).tobytes())


@pytest.mark.parametrize("n", sorted(RECORDED))
def test_recorded_results(pb2lib, n):
    import torch
    from pirate_b200.sifter import PATCH_LEN
    rng = np.random.default_rng(n)
    s = _sifter(rng)
    x = torch.from_numpy(rng.standard_normal((n, PATCH_LEN)).astype(np.float16)).cuda()
    y = torch.from_numpy((rng.random(n) < 0.5).astype(np.float32)).cuda()
    got = [_crc(s.forward(x).cpu().numpy())]
    loss, g = s.gradients(x, y)
    got += [_crc(np.array([loss], np.float32)), _crc(g)]
    losses = [s.train_step(x, y, 1e-3) for _ in range(3)]
    got += [_crc(np.array(losses, np.float32)), _crc(s.get_params())]
    assert tuple(got) == RECORDED[n]


def test_score_does_not_depend_on_the_batch(pb2lib):
    import torch
    from pirate_b200.sifter import PATCH_LEN
    rng = np.random.default_rng(5)
    s = _sifter(rng)
    x = torch.from_numpy(rng.standard_normal((1024, PATCH_LEN)).astype(np.float16)).cuda()
    whole = s.forward(x)
    for step in (8, 60, 100, 250, 512):
        parts = torch.cat([s.forward(x[i:i + step]) for i in range(0, 1024, step)])
        assert torch.equal(parts, whole), step
