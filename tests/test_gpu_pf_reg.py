"""The register peak finder at the edges of its geometry: every output time downsampling from 2 to 64, widths 1 to
32, chunks with fewer output times than a warp has lanes (coarse dms share warps) and partial tiles, subbands with
weights of their own; weights that are all positive (the largest profile value decides), and weights with zeros and
negative values (every product is compared); samples that are infinite or NaN. float32 outputs and tokens must equal
the fp32 oracle's bit for bit; with 16-bit rows, whose lanes share 16-byte pieces and words, those of the general kernel."""

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu

# (rank, nt, subbands, primary trees as (early triggers, max width, time downsampling))
CASES = [
    (6, 128, [1], [(0, 32, 2)]),                               # 32 halo lanes
    (6, 192, [1, 1], [(0, 16, 4), (0, 32, 4)]),                # 8 and 16 halo lanes, partial tiles
    (7, 64, [2, 1, 1], [(0, 8, 8), (0, 1, 4)]),                # 8 output times: four coarse dms per warp
    (7, 512, [0, 1], [(0, 32, 64), (0, 4, 32), (0, 2, 16)]),   # 8, 8 and 8 output times
    (8, 704, [0, 2, 1], [(1, 32, 16), (0, 32, 8)]),            # 44 output times: a full and a partial tile
]


@pytest.mark.parametrize("weights", ["positive", "signed"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "r%d_t%d" % (c[0], c[1]))
def test_pf_geometry_bitwise(pb2lib, case, weights):
    rank, nt, sb, pts = case
    prim = []
    for ip, (net, w, tds) in enumerate(pts):
        prim.append(dict(num_early_triggers=net, max_width=w, dm_downsampling=0, time_downsampling=tds,
                         wt_dm_downsampling=2 ** ((rank - (1 if ip else 0) - net + 1) // 2), wt_time_downsampling=max(16, tds)))
    cfg = H.toy_config(rank=rank, nfreq=2 ** rank // 2, nt=nt, subbands=sb, beams_per_gpu=2, beams_per_batch=2,
                       primary_trees=prim)
    nchunks = 4
    xs = H.make_inputs(cfg, nchunks, seed=rank + nt)
    if weights == "signed":
        xs[1][0, :, 17] = np.inf
        xs[2][1, 3, 40:44] = np.nan
    orc, _ = H.run_oracle(cfg, xs[:0], [])
    rng = np.random.default_rng(rank)
    ws = H.make_weights(orc, seed=rank, kind="bare" if weights == "positive" else "random")
    for w in ws:
        if weights == "positive":
            w *= rng.uniform(0.5, 2.0, w.shape).astype(np.float32)
        else:
            w *= rng.choice([1.0, 1.0, -1.0], w.shape).astype(np.float32)
    _, ores = H.run_oracle(cfg, xs, ws, 1, 32)
    _, _, gres = H.run_gpu(pb2lib, cfg, xs, ws)
    for seq in range(nchunks):
        for i in range(orc.ntrees):
            assert np.array_equal(gres[seq][0][i], ores[seq][0][i]), "out_max, chunk %d tree %d" % (seq, i)
            assert np.array_equal(gres[seq][1][i], ores[seq][1][i]), "out_argmax, chunk %d tree %d" % (seq, i)


CASES_16BIT = [
    (6, 128, [1], [(0, 32, 2)]),                               # 4 bytes per lane, 32 halo lanes
    (6, 320, [1], [(0, 4, 2)]),                                # 4 bytes per lane, 160 output times
    (6, 384, [1, 1], [(0, 16, 4), (0, 32, 4)]),                # 8 bytes per lane, 96 and 48 output times
    (7, 128, [2, 1, 1], [(0, 8, 16), (0, 1, 8)]),              # 8 output times: four coarse dms per warp
    (7, 512, [0, 1], [(0, 32, 64), (0, 4, 32), (0, 2, 16)]),   # 8, 8 and 8 output times
    (8, 768, [0, 2, 1], [(1, 32, 16), (0, 32, 8)]),            # 48 output times: a full and a partial tile
]


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("weights", ["positive", "signed"])
@pytest.mark.parametrize("case", CASES_16BIT, ids=lambda c: "r%d_t%d" % (c[0], c[1]))
def test_pf_geometry_16bit_same_as_general_kernel(pb2lib, case, weights, dtype):
    import torch
    rank, nt, sb, pts = case
    prim = []
    for ip, (net, w, tds) in enumerate(pts):
        prim.append(dict(num_early_triggers=net, max_width=w, dm_downsampling=0, time_downsampling=tds,
                         wt_dm_downsampling=2 ** ((rank - (1 if ip else 0) - net + 1) // 2), wt_time_downsampling=max(16, tds)))
    cfg = H.toy_config(rank=rank, nfreq=2 ** rank // 2, nt=nt, dtype=dtype, subbands=sb, beams_per_gpu=2, beams_per_batch=2,
                       primary_trees=prim)
    nchunks = 4
    xs = H.make_inputs(cfg, nchunks, seed=rank + nt)
    if weights == "signed":
        xs[1][0, :, 17] = np.inf
        xs[2][1, 3, 40:44] = np.nan
    orc, _ = H.run_oracle(cfg, xs[:0], [])
    rng = np.random.default_rng(rank)
    ws = H.make_weights(orc, seed=rank, kind="bare" if weights == "positive" else "random")
    bd = pb2lib.BatchedDedisperser([pb2lib.DedispersionPlan(pb2lib.DedispersionConfig.from_dict(cfg))], cuda_device_id=0)
    bd.allocate()
    for i, w in enumerate(ws):
        if weights == "positive":
            w *= rng.uniform(0.5, 2.0, w.shape).astype(np.float32)
        else:
            w *= rng.choice([1.0, 1.0, -1.0, 0.0], w.shape).astype(np.float32)
        bd.fill_all_weights(0, i, w)
    res = []
    for general in (True, False):
        bd.set_schedule([True], [general], [128])
        bd.reset()
        outs = []
        for x in xs:
            bd.input(0).copy_(torch.from_numpy(x).to(bd.device))
            bd.step()
            o = bd.outputs(0)
            outs += [t.clone() for t in o.out_max + o.out_argmax]
        torch.cuda.synchronize()
        res.append(outs)
    for a, b in zip(*res):
        assert torch.equal(a, b)
