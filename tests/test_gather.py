"""Rows of every residue of 4 (the gather takes 4, 2 or 1 columns a thread):
read lengths and row pitches around them, plain and packed, against the CPU
oracle, byte for byte."""
import dataclasses

import numpy as np
import pytest

from gsnp_gb300 import api, synth

from oracle_run import first_diff, flags_for, oracle_outputs


@pytest.mark.gpu
@pytest.mark.parametrize("L,pitch", [(48, 48), (49, 49), (50, 50), (50, 51), (50, 52), (48, 50), (49, 52), (250, 250),
                                     (2, 2), (1, 2), (254, 254)])
def test_rows_of_any_width(L, pitch, tmp_path, oracle_bin, native_lib):
    rng = np.random.default_rng(1000 * L + pitch)
    G, R = 5003, 6 * 5003 // L
    code = rng.integers(0, 4, G)
    acgt = np.frombuffer(b"ACTG", dtype=np.uint8)
    pos = np.sort(rng.integers(0, G - L - 1, R))
    length = rng.integers((L + 1) // 2, L + 1, R)
    cols = np.arange(L)[None, :]
    valid = cols < length[:, None]
    obs = np.where(rng.random((R, L)) < 0.02, rng.integers(0, 4, (R, L)), code[np.minimum(pos[:, None] + cols, G - 1)])
    seq = np.where(valid, acgt[obs], 0).astype(np.uint8)
    qual = np.where(valid, 64 + rng.integers(2, 41, (R, L)), 0).astype(np.uint8)
    none = np.zeros(0, dtype=np.int64)
    cfg = dataclasses.replace(synth.CONFIGS["c1"], name="rows", genome_len=G, read_lens=[L],
                              flags=["-L", str(L), "-t", "-u"])
    w = synth.Workload(config=cfg, seed=0, chr_name="chr1", ref=acgt[code], read_length=L, pos=pos.astype(np.int32),
                       length=length.astype(np.int32), hit=np.where(rng.random(R) < 0.05, 3, 1).astype(np.int32),
                       strand=np.where(rng.random(R) < 0.5, ord("-"), ord("+")).astype(np.uint8), seq=seq, qual=qual,
                       mismatch=np.zeros(R, dtype=np.int32), db_pos=none, db_hapmap=none.astype(np.uint8),
                       db_validated=none.astype(np.uint8), db_freq=np.zeros((0, 4)))
    flags = flags_for(w, synth.write_inputs(w, str(tmp_path)))
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    c, _, _ = api.run_workload(w, flags, precision=api.PRECISION_FP32_FIXUP)
    try:
        wide = np.zeros((2, R, pitch), dtype=np.uint8)
        wide[0, :, :L], wide[1, :, :L] = seq, qual
        q_min = api.params_from_flags(flags).q_min
        packed = api.pack_reads(wide[0], wide[1], w.length, q_min)
        for reads in (api.Caller.reads_struct(w.pos, w.length, w.hit, w.strand, wide[0], wide[1]),
                      api.Caller.reads_struct(w.pos, w.length, w.hit, w.strand, None, None, packed=packed,
                                              packed_qmin=q_min)):
            c.call(reads)
            got = c.format_cns(w.chr_name)
            if got != ref["cns"]:
                i, x, y = first_diff(got, ref["cns"])
                pytest.fail(f"L {L}, pitch {pitch}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")
    finally:
        c.close()
