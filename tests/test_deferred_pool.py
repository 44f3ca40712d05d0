"""A call that defers more records than its pool holds: the pass over the
deferred sites does nothing, the pool is grown and the call made again.  Dense
heterozygous sites at 300 reads ask for four million record words, where a new
context's pool holds three and as many sites as there are; in one segment,
several, and chunk by chunk, against the CPU oracle."""
import dataclasses

import numpy as np
import pytest

from gsnp_gb300 import api, synth

from oracle_run import first_diff, flags_for, oracle_outputs

WINDOW = 262144
POOL_WORDS = 48 * 65536   # of a new context


def het_workload() -> synth.Workload:
    rng = np.random.default_rng(5)
    L, G = 100, 2 * WINDOW + 60013
    code = rng.integers(0, 4, G)
    starts = np.sort(np.concatenate([lo + rng.integers(0, n, 3 * n) for lo, n in
                                     ((5000, 2000), (WINDOW + 1000, 40000), (2 * WINDOW + 30000, 2000))]))
    R = starts.size
    minus = rng.random(R) < 0.5
    hap = np.stack([code, np.where(rng.random(G) < 0.5, (code + 1 + rng.integers(0, 3, G)) % 4, code)])
    site = starts[:, None] + np.arange(L)[None, :]
    q = np.clip(np.rint(rng.normal(30, 8, (R, L))), 2, 40).astype(np.int64)
    truth = hap[rng.integers(0, 2, R)[:, None], site]
    obs = np.where(rng.random((R, L)) < 10.0 ** (-q / 10.0), (truth + rng.integers(1, 4, (R, L))) % 4, truth)
    cfg = dataclasses.replace(synth.CONFIGS["c1"], name="hets", genome_len=G, read_lens=[L],
                              flags=["-L", str(L), "-t", "-u"])
    none = np.zeros(0, dtype=np.int64)
    acgt = np.frombuffer(b"ACTG", dtype=np.uint8)
    return synth.Workload(config=cfg, seed=0, chr_name="chr1", ref=acgt[code], read_length=L,
                          pos=starts.astype(np.int32), length=np.full(R, L, dtype=np.int32),
                          hit=np.ones(R, dtype=np.int32),
                          strand=np.where(minus, ord("-"), ord("+")).astype(np.uint8), seq=acgt[obs],
                          qual=(64 + q).astype(np.uint8), mismatch=np.zeros(R, dtype=np.int32), db_pos=none,
                          db_hapmap=none.astype(np.uint8), db_validated=none.astype(np.uint8),
                          db_freq=np.zeros((0, 4)))


@pytest.fixture(scope="module")
def expected(tmp_path_factory, oracle_bin):
    w = het_workload()
    d = str(tmp_path_factory.mktemp("hets"))
    paths = synth.write_inputs(w, d)
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, d)
    assert ref["rc"] == 0, ref["stderr"]
    return w, flags, ref["cns"]


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["one", "segments", "streamed"])
def test_pool_grown_and_call_redone(how, expected, tmp_path, native_lib, monkeypatch):
    w, flags, want = expected
    monkeypatch.setenv("GSNP_SEGMENTS", "3" if how == "segments" else "1")
    p = api.params_from_flags(flags, api.PRECISION_FP32_FIXUP)
    arrs = [np.ascontiguousarray(x) for x in (w.pos, w.length, w.hit, w.strand, w.seq, w.qual)]
    reads = api.Caller.reads_struct(*arrs)
    with api.Caller() as c:
        c.load_reference(api.site_codes(w.ref))
        c.load_tables(p, c.calibrate(p, reads), c.prior_table(p), c.rank_table())
        out = np.zeros(w.genome_len, dtype=api.SITE_DTYPE)
        if how == "streamed":
            c.set_option("stream_windows", 1)
            c.call_streamed(reads, w.chr_name, out.ctypes.data, str(tmp_path / "cns"))
            got = (tmp_path / "cns").read_bytes()
        else:
            c.call_into(reads, out.ctypes.data)
            got = c.format_cns(w.chr_name)
            assert out.tobytes() == c.fetch().tobytes()
        # nearly all of them hold 255 records
        assert c.stats()["deferred_sites"] * 240 > POOL_WORDS
        assert c.stats()["sample_mismatches"] == 0
    if got != want:
        i, x, y = first_diff(got, want)
        pytest.fail(f"{how}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")
