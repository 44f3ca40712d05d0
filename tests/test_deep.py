"""Columns of hundreds of records (a warp takes a site there) against the CPU
oracle, byte for byte: depths around the 128- and 255-record lines, a genome
that ends within a tile, heterozygous sites whose rank sums are taken, short
reads whose records share cycles, and deep sites in a window whose likelihood
and counts a later window without reads shows."""
import dataclasses

import numpy as np
import pytest

from gsnp_gb300 import api, synth

from oracle_run import first_diff, flags_for, oracle_outputs

WINDOW = 262144


def deep_workload(kind: str) -> synth.Workload:
    rng = np.random.default_rng(sum(map(ord, kind)))
    L = 20 if kind == "short" else 100
    G = 4 * WINDOW + 13 if kind == "gap" else 4013
    code = rng.integers(0, 4, G)
    depths = [100, 127, 128, 129, 130, 200, 254, 255, 256, 257, 400]
    first = [WINDOW - 4100, 3 * WINDOW + 40000] if kind == "gap" else [50]
    starts = np.concatenate([np.full(d, f + 350 * k) + rng.integers(0, 5 if kind == "short" else 60, d)
                             for f in first for k, d in enumerate(depths)])
    if kind == "end":
        starts = np.concatenate([starts, G - L - 1 - rng.integers(0, 40, 300)])
    starts = np.sort(starts)
    R = starts.size
    length = np.where(rng.random(R) < 0.2, rng.integers(L // 2, L + 1, R), L)
    minus = rng.random(R) < 0.5
    hit = np.where(rng.random(R) < 0.05, rng.integers(2, 9, R), 1).astype(np.int32)
    hap = np.stack([code, np.where(rng.random(G) < 0.05, (code + 1 + rng.integers(0, 3, G)) % 4, code)])
    cols = np.arange(L)[None, :]
    valid = cols < length[:, None]
    site = np.minimum(starts[:, None] + cols, G - 1)
    q = np.clip(np.rint(rng.normal(30, 8, (R, L))), 2, 40).astype(np.int64)
    truth = np.take_along_axis(hap[rng.integers(0, 2, R)], site, axis=1)
    obs = np.where(rng.random((R, L)) < 10.0 ** (-q / 10.0), (truth + rng.integers(1, 4, (R, L))) % 4, truth)
    cfg = dataclasses.replace(synth.CONFIGS["c1"], name="deep", genome_len=G, read_lens=[L],
                              flags=["-L", str(L), "-t", "-u"])
    none = np.zeros(0, dtype=np.int64)
    acgt = np.frombuffer(b"ACTG", dtype=np.uint8)
    return synth.Workload(config=cfg, seed=0, chr_name="chr1", ref=acgt[code], read_length=L,
                          pos=starts.astype(np.int32), length=length.astype(np.int32), hit=hit,
                          strand=np.where(minus, ord("-"), ord("+")).astype(np.uint8),
                          seq=np.where(valid, acgt[obs], 0).astype(np.uint8),
                          qual=np.where(valid, 64 + q, 0).astype(np.uint8), mismatch=np.zeros(R, dtype=np.int32),
                          db_pos=none, db_hapmap=none.astype(np.uint8), db_validated=none.astype(np.uint8),
                          db_freq=np.zeros((0, 4)))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "end", "short", "gap"])
def test_deep_columns_match_oracle(kind, tmp_path, oracle_bin, native_lib):
    w = deep_workload(kind)
    paths = synth.write_inputs(w, str(tmp_path))
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    for prec in (api.PRECISION_FP64, api.PRECISION_FP32_FIXUP):
        c, _, _ = api.run_workload(w, flags, precision=prec)
        try:
            got = c.format_cns(w.chr_name)
            slots = [launch["slots"] for launch in c.last_launches() if launch["tiles"]]
        finally:
            c.close()
        assert 256 in slots
        if got != ref["cns"]:
            i, x, y = first_diff(got, ref["cns"])
            pytest.fail(f"{kind}, precision {prec}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "gap"])
def test_deep_columns_with_spilling_qualities(kind, tmp_path, oracle_bin, native_lib):
    """Qualities whose record lies under another base than the read's: a score
    of 0 or above 64 spills into the record word's base, as in the reference.
    A deep site's terms, and the likelihood a later window takes from it, go by
    the record's base; its counts go by the read's."""
    w = deep_workload(kind)
    rng = np.random.default_rng(17)
    odd = rng.random(w.qual.shape)
    q = w.qual.astype(np.int64) - 64
    q = np.where(odd < 0.02, 0, np.where(odd < 0.05, rng.integers(63, 67, w.qual.shape), q))
    w.qual = np.where(w.qual > 0, 33 + q, 0).astype(np.uint8)
    w.config = dataclasses.replace(w.config, flags=w.config.flags + ["-z", "!", "-Q", "d"])
    paths = synth.write_inputs(w, str(tmp_path))
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    for prec in (api.PRECISION_FP64, api.PRECISION_FP32_FIXUP):
        c, _, _ = api.run_workload(w, flags, precision=prec)
        try:
            got = c.format_cns(w.chr_name)
            slots = [launch["slots"] for launch in c.last_launches() if launch["tiles"]]
        finally:
            c.close()
        assert 256 in slots
        if got != ref["cns"]:
            i, x, y = first_diff(got, ref["cns"])
            pytest.fail(f"{kind}, precision {prec}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")
