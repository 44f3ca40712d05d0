"""The short form of the calling kernels' sites (gsnp_gb300/csrc/lean.cuh).

CPU: its sort, walk and proof, compiled for the host, against the general walk
and the FP64 posterior (tests/native/lean_check.cpp).

GPU: both forms against the oracle on alignments made to sit at its edges and
on either side of the line to the general form: depths around its record slots,
more repeated (strand, cycle) keys than its counts hold, qualities outside
1 .. 63, reads of several hits, reads of length 1 to 255, and a genome that ends
inside a tile.  The bytes of the cns text must be the same."""
import dataclasses
import os
import subprocess

import numpy as np
import pytest

from gsnp_gb300 import api, synth

from oracle_run import first_diff, flags_for, oracle_outputs

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lean_check(tmp_path_factory):
    from gsnp_gb300 import build
    exe = str(tmp_path_factory.mktemp("lean") / "lean_check")
    csrc = os.path.join(ROOT, "gsnp_gb300", "csrc")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I" + csrc,
                        "-I" + os.path.join(ROOT, "include"), "-I" + build._cuda_include(),
                        os.path.join(ROOT, "tests", "native", "lean_check.cpp"),
                        os.path.join(csrc, "tables.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.mark.parametrize("sites,seed,length", [(200000, 1, 100), (60000, 2, 255), (60000, 3, 35)])
def test_lean_decisions_equal_fp64(sites, seed, length, lean_check):
    r = subprocess.run([lean_check, str(sites), str(seed), str(length)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    words = r.stdout.split()
    decided, hom = int(words[words.index("decided") + 1]), int(words[words.index("of") + 1])
    decided64 = int(words[words.index("decided64") + 1])
    assert decided > hom * 9 // 10 and decided64 > hom * 9 // 10, r.stdout   # not vacuous


def edge_workload(kind: str) -> synth.Workload:
    """A genome of 4,013 sites and alignments of the given kind."""
    rng = np.random.default_rng(sum(map(ord, kind)))
    G = 4013
    L = 255 if kind == "lengths" else 100
    code = rng.integers(0, 4, G)
    ref = np.frombuffer(b"ACTG", dtype=np.uint8)[code]
    if kind in ("slots", "deep_slots"):
        # one depth per 200-site stretch: exactly d reads over each of its inner sites
        depths = [16, 17, 31, 32, 33, 40, 41] if kind == "slots" else [47, 48, 49, 63, 64, 65, 66]
        starts = np.concatenate([np.full(d, 200 + 500 * k) + rng.integers(0, 60, d) for k, d in enumerate(depths)])
        length = np.full(starts.size, 100)
    elif kind == "repeats":
        # from few to many reads sharing a start, and many starts shared by two
        starts = np.concatenate([np.full(n, 200 + 220 * k) for k, n in enumerate([2, 3, 14, 15, 16, 17, 30])] +
                                [np.repeat(2400 + 3 * np.arange(n) + 250 * k, 2) for k, n in
                                 enumerate([7, 8, 15, 16, 20])])
        length = np.full(starts.size, 100)
    elif kind == "lengths":
        length = rng.integers(1, 256, 900)
        starts = rng.integers(0, G - 256, 900)
    else:
        starts = rng.integers(0, G - 101, 1100)
        length = np.full(starts.size, 100)
    order = np.argsort(starts, kind="stable")
    starts, length = starts[order], length[order]
    R = starts.size
    minus = starts % 2 == 1 if kind == "repeats" else rng.random(R) < 0.5   # reads that start together: one strand
    hit = np.where(rng.random(R) < (0.5 if kind == "hits" else 0.05), rng.integers(2, 9, R), 1).astype(np.int32)
    hap = np.stack([code, np.where(rng.random(G) < 0.01, (code + 1 + rng.integers(0, 3, G)) % 4, code)])
    cols = np.arange(L)[None, :]
    valid = cols < length[:, None]
    site = np.minimum(starts[:, None] + cols, G - 1)
    q = np.clip(np.rint(rng.normal(30, 8, (R, L))), 2, 40).astype(np.int64)
    if kind == "qualities":
        odd = rng.random((R, L))
        q = np.where(odd < 0.02, 0, np.where(odd < 0.04, 63, np.where(odd < 0.05, -1, q)))
    if kind == "wide":
        q = np.where(rng.random((R, L)) < 0.01, rng.integers(41, 62, (R, L)), q)
    truth = np.take_along_axis(hap[rng.integers(0, 2, R)], site, axis=1)
    err = rng.random((R, L)) < 10.0 ** (-np.maximum(q, 1) / 10.0)
    obs = np.where(err, (truth + rng.integers(1, 4, (R, L))) % 4, truth)
    seq = np.where(valid, np.frombuffer(b"ACTG", dtype=np.uint8)[obs], 0).astype(np.uint8)
    qual = np.where(valid, 64 + q, 0).astype(np.uint8)
    cfg = dataclasses.replace(synth.CONFIGS["c1"], name="edge", genome_len=G, read_lens=[L],
                              flags=["-L", str(L), "-t", "-u"] + (["-Q", "\x7f"] if kind in ("wide", "qualities") else []))
    none = np.zeros(0, dtype=np.int64)
    return synth.Workload(config=cfg, seed=0, chr_name="chr1", ref=ref, read_length=L, pos=starts.astype(np.int32),
                          length=length.astype(np.int32), hit=hit, strand=np.where(minus, ord("-"), ord("+")).astype(np.uint8),
                          seq=seq, qual=qual, mismatch=np.zeros(R, dtype=np.int32), db_pos=none,
                          db_hapmap=none.astype(np.uint8), db_validated=none.astype(np.uint8),
                          db_freq=np.zeros((0, 4)))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["plain", "slots", "deep_slots", "repeats", "lengths", "hits", "wide", "qualities"])
def test_edges_match_oracle(kind, tmp_path, oracle_bin, native_lib):
    w = edge_workload(kind)
    paths = synth.write_inputs(w, str(tmp_path))
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    for prec in (api.PRECISION_FP64, api.PRECISION_FP32_FIXUP):
        c, _, _ = api.run_workload(w, flags, precision=prec)
        try:
            got = c.format_cns(w.chr_name)
            assert c.stats()["sample_mismatches"] == 0
        finally:
            c.close()
        if got != ref["cns"]:
            i, x, y = first_diff(got, ref["cns"])
            pytest.fail(f"{kind}, precision {prec}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")


@pytest.mark.gpu
def test_recall_under_another_qmin(native_lib):
    """Tables loaded with another q_min after a call: the recalled sites are
    those of a call made under it (the resident elements count from q_min)."""
    w = edge_workload("plain")
    flags = list(w.config.flags)
    got = {}
    for recall in (False, True):
        c, reads, pm = api.run_workload(w, flags, precision=api.PRECISION_FP32_FIXUP)
        try:
            p = api.params_from_flags(flags + ["-z", "D", "-Q", "h"], api.PRECISION_FP32_FIXUP)
            c.load_tables(p, pm, c.prior_table(p), c.rank_table())
            if recall:
                c.recall_resident()
            else:
                c.call(reads)
            got[recall] = c.fetch()
        finally:
            c.close()
    assert got[True].tobytes() == got[False].tobytes()


def test_short_form_needs_terms_of_zero_or_less(tmp_path):
    """A matrix entry above 1 gives a positive term, for which the FP32 bounds
    that choose the second genotype do not hold."""
    from gsnp_gb300 import build
    exe = str(tmp_path / "lean_rules_check")
    csrc = os.path.join(ROOT, "gsnp_gb300", "csrc")
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-I" + csrc,
                        "-I" + os.path.join(ROOT, "include"), "-I" + build._cuda_include(),
                        os.path.join(ROOT, "tests", "native", "lean_rules_check.cpp"),
                        os.path.join(csrc, "tables.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.split("\n")[:3] == ["plain lean 1", "above lean 0", "unreached lean 1"], r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32_FIXUP])
def test_matrix_entry_above_one_takes_the_general_form(precision, native_lib):
    """Either form then runs the binned FP64 kernels, whatever "persistent" says."""
    w = edge_workload("plain")
    c, reads, pm = api.run_workload(w, list(w.config.flags), precision=precision)
    try:
        assert 4 in [launch["kind"] for launch in c.last_launches()]
        p = api.params_from_flags(w.config.flags, precision)
        pm = pm.copy()
        pm[30 << 12 | 50 << 4 | 5] = 1.2
        c.load_tables(p, pm, c.prior_table(p), c.rank_table())
        got = {}
        for persistent in (1, 0):
            c.set_option("persistent", persistent)
            c.call(reads)
            got[persistent] = c.fetch().tobytes()
            assert {launch["kind"] for launch in c.last_launches() if launch["tiles"]} <= {0, 1}
        assert got[0] == got[1]
    finally:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32_FIXUP])
def test_qualities_zero_and_64_stay_in_the_short_form(precision, tmp_path, oracle_bin, native_lib):
    """Records of quality 0, whose word lies under another base, and of 64: no
    tile is left to the binned kernels, and the text is the oracle's."""
    w = edge_workload("plain")
    odd = np.random.default_rng(3).random(w.qual.shape)
    q = w.qual.astype(np.int64) - 64
    q = np.where(odd < 0.05, 0, np.where(odd < 0.08, 64, q))
    w.qual = np.where(w.qual > 0, 33 + q, 0).astype(np.uint8)
    w.config = dataclasses.replace(w.config, flags=w.config.flags + ["-z", "!", "-Q", "d"])
    paths = synth.write_inputs(w, str(tmp_path))
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    c, _, _ = api.run_workload(w, flags, precision=precision)
    try:
        got = c.format_cns(w.chr_name)
        left = sum(launch["tiles"] for launch in c.last_launches() if launch["kind"] in (1, 2, 6))
        assert c.stats()["sample_mismatches"] == 0
    finally:
        c.close()
    if got != ref["cns"]:
        i, x, y = first_diff(got, ref["cns"])
        pytest.fail(f"precision {precision}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")
    assert left == 0


@pytest.mark.gpu
@pytest.mark.parametrize("sites,slots", [(30013, 64), (1200013, 48)])
def test_tiles_it_can_never_take_go_to_one_shallow_bin(sites, slots, tmp_path, oracle_bin, native_lib, monkeypatch):
    """Twenty reads of one start and strand everywhere: no tile of the short form
    but too deep for none of its slots.  A segment of many times the tiles that the
    64-slot kernel holds at once gives them to the 48-slot one."""
    monkeypatch.setenv("GSNP_SEGMENTS", "1")
    w = edge_workload("plain")
    rng = np.random.default_rng(9)
    L, code = 100, rng.integers(0, 4, sites)
    acgt = np.frombuffer(b"ACTG", dtype=np.uint8)
    pos = np.repeat(np.arange(0, sites - L - 1, L), 20)
    R = pos.size
    base = code[pos[:, None] + np.arange(L)]
    seq = acgt[np.where(rng.random((R, L)) < 0.01, rng.integers(0, 4, (R, L)), base)]
    w = dataclasses.replace(w, ref=acgt[code], config=dataclasses.replace(w.config, genome_len=sites),
                            pos=pos.astype(np.int32), length=np.full(R, L, dtype=np.int32),
                            hit=np.ones(R, dtype=np.int32),
                            strand=np.where(pos // L % 2 == 0, ord("+"), ord("-")).astype(np.uint8), seq=seq,
                            qual=(64 + rng.integers(2, 41, (R, L))).astype(np.uint8),
                            mismatch=np.zeros(R, dtype=np.int32))
    paths = synth.write_inputs(w, str(tmp_path))
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    for prec in (api.PRECISION_FP64, api.PRECISION_FP32_FIXUP):
        c, _, _ = api.run_workload(w, flags, precision=prec)
        try:
            got = c.format_cns(w.chr_name)
            bins = {launch["slots"] for launch in c.last_launches() if launch["kind"] in (1, 2, 6) and launch["tiles"]}
        finally:
            c.close()
        if got != ref["cns"]:
            i, x, y = first_diff(got, ref["cns"])
            pytest.fail(f"{sites}, precision {prec}: first differing row {i}:\n gpu   : {x!r}\n oracle: {y!r}")
        assert bins == {slots}
