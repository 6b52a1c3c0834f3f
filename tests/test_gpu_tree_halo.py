"""The tree kernels at the edges of their tiles: float32 outputs must equal the fp32 oracle's bit for bit.

Tiles are 64 samples at dd ranks 7 and 8, 128 at 6 and 256 below, the last one of a chunk what remains; segments
512-2048 samples; blocks read their rows at every alignment. The cases take chunks of one short tile, with a short
last tile, longer than a segment, every dd rank from 1 to 8, full-band and (staggered) subband outputs."""

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu

# (rank, nt, subbands, primary trees as (early triggers, max width), chunks)
CASES = [
    (3, 32, [1], [(0, 4)], 9),                         # dd ranks 1 + 2, one tile of 32 samples
    (4, 96, [0, 1], [(1, 4)], 7),                      # dd ranks 2 + 1, 2; one tile of 96
    (5, 352, [1, 1], [(2, 8)], 4),                     # dd ranks 2 + 1..3; a tile and 96 samples
    (6, 4160, [0, 0, 1], [(1, 8), (0, 4)], 2),         # two segments of 2048 and 64 samples
    (9, 2560, [0, 0, 0, 1], [(0, 16), (0, 8)], 2),     # dd ranks 4, 5: a segment and a quarter
    (10, 448, [4, 7, 3, 1], [(1, 8)], 4),              # every subband level, staggered pairs
    (12, 192, [0, 3, 0, 1], [(1, 16), (0, 8)], 4),     # dd ranks 5, 6; a tile and a half
    (14, 640, [0, 0, 0, 0, 1], [(0, 8), (0, 4)], 2),   # dd rank 7: ten tiles
    (14, 2144, [0, 0, 0, 0, 1], [(0, 8)], 2),          # dd rank 7: a float32 segment (2048), a tile and a half
    (16, 1088, [0, 1, 0, 0, 1], [(0, 8)], 2),          # dd rank 8: a float32 segment (1024) and one tile
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "r%d_t%d" % (c[0], c[1]))
def test_tree_tiles_bitwise(pb2lib, case):
    rank, nt, sb, pts, nchunks = case
    prim = []
    for ip, (net, w) in enumerate(pts):
        prim.append(dict(num_early_triggers=net, max_width=w, dm_downsampling=0, time_downsampling=0,
                         wt_dm_downsampling=2 ** ((rank - (1 if ip else 0) - net + 1) // 2), wt_time_downsampling=16))
    cfg = H.toy_config(rank=rank, nfreq=max(8, 2 ** rank // 3), nt=nt, subbands=sb, beams_per_gpu=1, beams_per_batch=1,
                       primary_trees=prim)
    xs = H.make_inputs(cfg, nchunks, seed=rank + nt)
    orc, _ = H.run_oracle(cfg, xs[:0], [])
    ws = H.make_weights(orc, seed=rank)
    _, ores = H.run_oracle(cfg, xs, ws, 1, 32)
    _, _, gres = H.run_gpu(pb2lib, cfg, xs, ws)
    for seq in range(nchunks):
        for i in range(orc.ntrees):
            assert np.array_equal(gres[seq][0][i], ores[seq][0][i]), "out_max, chunk %d tree %d" % (seq, i)
            assert np.array_equal(gres[seq][1][i], ores[seq][1][i]), "out_argmax, chunk %d tree %d" % (seq, i)


@pytest.mark.parametrize("dtype,tol", [("float16", 1e-2), ("bfloat16", 6e-2)])
def test_tree_tiles_16bit(pb2lib, dtype, tol):
    """16-bit rows start at any sample of a 16-byte chunk; against the FP64 oracle, in sigma (bare weights)."""
    cfg = H.toy_config(rank=13, nfreq=3000, nt=192, dtype=dtype, subbands=[0, 3, 0, 1], beams_per_gpu=1, beams_per_batch=1,
                       primary_trees=[dict(num_early_triggers=1, max_width=8, dm_downsampling=0, time_downsampling=0,
                                           wt_dm_downsampling=64, wt_time_downsampling=16)])
    xs = H.make_inputs(cfg, 4, seed=3)
    orc, _ = H.run_oracle(cfg, xs[:0], [])
    ws = H.make_weights(orc, seed=3, kind="bare")
    _, ores = H.run_oracle(cfg, xs, ws, 1, 64)
    _, _, gres = H.run_gpu(pb2lib, cfg, xs, ws)
    for seq in range(4):
        for i in range(orc.ntrees):
            assert np.abs(gres[seq][0][i] - ores[seq][0][i]).max() <= tol


def test_delay_lines_need_no_whole_chunks(pb2lib):
    """Delay lines hold a multiple of 32 samples at every chunk length: 64 samples more per chunk cost 64/2048 more
    memory, also where the chunk is then no multiple of the kernel's tile (128 samples at dd rank 6)."""
    size = {}
    for nt in (2048, 2112):
        cfg = H.toy_config(rank=12, nfreq=1024, nt=nt, dtype="float16", subbands=[0, 0, 0, 1], beams_per_gpu=1, beams_per_batch=1,
                           primary_trees=[dict(num_early_triggers=0, max_width=8, dm_downsampling=0, time_downsampling=0,
                                               wt_dm_downsampling=64, wt_time_downsampling=16)])
        dd = pb2lib.GpuDedisperser(pb2lib.DedispersionPlan(pb2lib.DedispersionConfig.from_dict(cfg)))
        dd.allocate()
        size[nt] = dd.device_bytes()
    assert size[2112] <= 1.04 * size[2048]


# (rank, subbands, samples per long chunk): dd ranks 4, 6, 7 and 8; past the 16-bit segments of 2048, 2048, 512 and 2048
# samples, the last tile partial at dd ranks 4 and 6.
@pytest.mark.parametrize("dtype", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("rank,subbands,nt", [(8, [1, 1, 1], 2112), (12, [0, 1, 0, 1], 2112), (14, [0, 0, 0, 0, 1], 576), (16, [0, 0, 0, 0, 1], 2112)])
def test_chunk_length_does_not_change_outputs(pb2lib, rank, subbands, nt, dtype):
    """A stream cut into long chunks gives what it gives cut into chunks of 64 samples, bit for bit."""
    rng = np.random.default_rng(rank)
    x = rng.standard_normal((1, 300, 2 * nt)).astype(np.float32)
    res = []
    for n in (64, nt):
        cfg = H.toy_config(rank=rank, nfreq=300, nt=n, dtype=dtype, subbands=subbands, beams_per_gpu=1, beams_per_batch=1,
                           primary_trees=[dict(num_early_triggers=0, max_width=8, dm_downsampling=0, time_downsampling=0,
                                               wt_dm_downsampling=2 ** (rank // 2), wt_time_downsampling=16)])
        orc, _ = H.run_oracle(cfg, [], [])
        ws = H.make_weights(orc, seed=1, kind="bare")
        _, _, g = H.run_gpu(pb2lib, cfg, [np.ascontiguousarray(x[:, :, k:k + n]) for k in range(0, 2 * nt, n)], ws)
        res.append([np.concatenate([r[k][0] for r in g], axis=-1) for k in (0, 1)])
    assert np.array_equal(res[0][0], res[1][0]) and np.array_equal(res[0][1], res[1][1])
