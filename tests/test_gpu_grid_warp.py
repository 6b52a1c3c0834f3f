"""Gridding and lagged downsampling by a warp per channel pair, at the edges: fewer pairs than a block has warps, chunks
of one step and of several, split over blocks or carried from step to step, 0 to 4 downsampled levels in 8- and 16-sample
windows, input channels per tree channel from a fraction to dozens, and int4 input with and without the tables. float32
outputs must equal the fp32 oracle's bit for bit; int4 input must give what the dequantized samples give; chunks that
the kernel does not take must give what the same stream gives in chunks that it takes."""

import numpy as np
import pytest

import helpers as H
import oracle as O

pytestmark = pytest.mark.gpu

# (rank, nfreq, nt, number of primary trees, beams)
CASES = [
    (2, 3, 256, 1, 2),       # 2 pairs, one step
    (7, 40, 768, 2, 1),      # 3 tree channels per input channel; every step in a block of its own
    (7, 350, 1280, 4, 1),    # levels of one sample per window
    (8, 120, 2048, 3, 8),    # two steps per block
    (6, 64, 1536, 5, 2),     # four levels: 16-sample windows
    (7, 3000, 512, 5, 1),    # 23 input channels per tree channel
]


def _cfg(rank, nfreq, nt, npri, beams, dtype="float32"):
    prim = [dict(num_early_triggers=0, max_width=4, dm_downsampling=0, time_downsampling=0,
                 wt_dm_downsampling=2 ** ((rank - (1 if i else 0) + 1) // 2), wt_time_downsampling=16) for i in range(npri)]
    return H.toy_config(rank=rank, nfreq=nfreq, nt=nt, dtype=dtype, subbands=[1], beams_per_gpu=beams, beams_per_batch=beams,
                        primary_trees=prim)


@pytest.mark.parametrize("case", CASES, ids=lambda c: "r%d_f%d_t%d_p%d" % c[:4])
def test_grid_warp_bitwise(pb2lib, case):
    cfg = _cfg(*case)
    xs = H.make_inputs(cfg, 3, seed=case[1])
    orc, _ = H.run_oracle(cfg, xs[:0], [])
    ws = H.make_weights(orc, seed=1, kind="bare")
    _, ores = H.run_oracle(cfg, xs, ws, 1, 32)
    _, _, gres = H.run_gpu(pb2lib, cfg, xs, ws)
    for seq in range(3):
        for i in range(orc.ntrees):
            assert np.array_equal(gres[seq][0][i], ores[seq][0][i]) and np.array_equal(gres[seq][1][i], ores[seq][1][i])


# Chunks of 256 and 768 samples (8-sample windows), 512 and 1024 (16-sample windows).
@pytest.mark.parametrize("nt,npri,nfreq", [(256, 3, 100), (512, 1, 40), (1024, 5, 100), (768, 3, 100), (512, 3, 1500)])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_grid_warp_int4(pb2lib, dtype, nt, npri, nfreq):
    import torch
    pb = pb2lib
    cfg = _cfg(8, nfreq, nt, npri, 2, dtype)
    d, so = O.random_quantized(np.random.default_rng(4), 2, nfreq, 3 * nt)
    res = []
    for int4 in (False, True):
        plan = pb.DedispersionPlan(pb.DedispersionConfig.from_dict(cfg))
        dd = pb.GpuDedisperser(plan, cuda_device_id=0, num_consumers=1)
        dd.allocate()
        dd.fill_analytic_weights(np.ones(nfreq))
        outs = []
        for c in range(3):
            dc = torch.from_numpy(np.ascontiguousarray(d[:, :, c * nt // 2:(c + 1) * nt // 2])).cuda()
            sc = torch.from_numpy(np.ascontiguousarray(so[:, :, c * nt // 256:(c + 1) * nt // 256])).cuda()
            if int4:
                with dd.get_input_int4() as (data, scoff):
                    data.copy_(dc)
                    scoff.copy_(sc)
            else:
                with dd.get_input() as arr:
                    pb.dequantize(arr, sc, dc)
            with dd.get_output(0, sync=True) as out:
                outs += [t.clone() for t in out.out_max + out.out_argmax]
        res.append(outs)
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("nfreq", [100, 256, 1500])   # up to 1 and 2, 2 to 3, and 2 to 17 input channels per tree channel
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
def test_grid_lds_same_as_grid_warp(pb2lib, dtype, nfreq):
    """A stream in chunks of 384 samples (a thread per window, with a downsampled level) and of 768 (a warp per pair)."""
    rng = np.random.default_rng(9)
    x = rng.standard_normal((2, nfreq, 4 * 768)).astype(np.float32)
    res = []
    for nt in (384, 768):
        cfg = _cfg(8, nfreq, nt, 2, 2, dtype)
        orc, _ = H.run_oracle(cfg, [], [])
        ws = H.make_weights(orc, seed=1, kind="bare")
        _, _, g = H.run_gpu(pb2lib, cfg, [np.ascontiguousarray(x[:, :, k:k + nt]) for k in range(0, x.shape[2], nt)], ws)
        res.append([np.concatenate([r[k][i] for r in g], axis=-1) for k in (0, 1) for i in range(orc.ntrees)])
    for a, b in zip(*res):
        assert np.array_equal(a, b)
