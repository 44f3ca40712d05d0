"""The GPU's -C files over more windows than a batch holds, most of them with a
handful of runs in every column (a few reads on a long genome), against the
host encoder, byte for byte."""
import dataclasses
import os

import numpy as np
import pytest

from gsnp_gb300 import api, synth

FILES = [".1_2", ".3_4_6", ".5_7_8_9_14_16", ".10", ".11_12_13", ".15_17"]


@pytest.mark.gpu
@pytest.mark.parametrize("reads", [60, 40000])
def test_files_of_several_batches(reads, tmp_path, native_lib):
    rng = np.random.default_rng(reads)
    G, L = 66 * 262144 + 1001, 100
    code = rng.integers(0, 4, G)
    acgt = np.frombuffer(b"ACTG", dtype=np.uint8)
    pos = np.sort(np.concatenate([np.arange(67) * 262144 % (G - L - 1), rng.integers(0, G - L - 1, reads)]))
    R = pos.size
    site = pos[:, None] + np.arange(L)[None, :]
    obs = np.where(rng.random((R, L)) < 0.02, rng.integers(0, 4, (R, L)), code[site])
    none = np.zeros(0, dtype=np.int64)
    cfg = dataclasses.replace(synth.CONFIGS["c1"], name="sparse", genome_len=G, read_lens=[L],
                              flags=["-L", str(L), "-t", "-u"])
    w = synth.Workload(config=cfg, seed=0, chr_name="chr1", ref=acgt[code], read_length=L, pos=pos.astype(np.int32),
                       length=np.full(R, L, dtype=np.int32), hit=np.ones(R, dtype=np.int32),
                       strand=np.where(rng.random(R) < 0.5, ord("-"), ord("+")).astype(np.uint8), seq=acgt[obs],
                       qual=(64 + rng.integers(2, 41, (R, L))).astype(np.uint8), mismatch=np.zeros(R, dtype=np.int32),
                       db_pos=none, db_hapmap=none.astype(np.uint8), db_validated=none.astype(np.uint8),
                       db_freq=np.zeros((0, 4)))
    c, _, _ = api.run_workload(w, w.config.flags, precision=api.PRECISION_FP32_FIXUP)
    try:
        out = {}
        for gpu in (1, 0):
            c.set_option("columns_gpu", gpu)
            base = str(tmp_path / ("gpu" if gpu else "host") / "cns")
            os.makedirs(os.path.dirname(base))
            assert c.lib.gsnp_write_columns(c.ctx, b"chr1", base.encode()) == 0, c.lib.gsnp_context_error(c.ctx)
            out[gpu] = {f: open(base + f, "rb").read() for f in FILES}
    finally:
        c.close()
    for f in FILES:
        assert out[1][f] == out[0][f], f"{f} differs between the GPU and host encoders"
