"""One context used for one chromosome after another, and with other tables in
between: what it keeps on the device has to fit each call, and the calls are
those of a context of their own."""
import dataclasses

import numpy as np
import pytest

from gsnp_gb300 import api

from test_lean import edge_workload


def arrays(w):
    return [np.ascontiguousarray(x) for x in (w.pos, w.length, w.hit, w.strand, w.seq, w.qual)]


def load(c, w, precision=api.PRECISION_FP32_FIXUP):
    """The workload's reference and tables into c; its alignments."""
    reads = api.Caller.reads_struct(*c.__dict__.setdefault("arrays", {}).setdefault(id(w), arrays(w)))
    p = api.params_from_flags(w.config.flags, precision)
    c.load_reference(api.site_codes(w.ref))
    c.load_tables(p, c.calibrate(p, reads), c.prior_table(p), c.rank_table())
    return reads


def own_context(w, precision=api.PRECISION_FP32_FIXUP):
    with api.Caller() as c:
        c.call(load(c, w, precision))
        return c.fetch().tobytes()


@pytest.mark.gpu
def test_longer_reads_after_more_reads(native_lib):
    """900 reads of up to 255 bases after 1,100 of 100: fewer rows, more of them in all."""
    short, long = edge_workload("plain"), edge_workload("lengths")
    assert len(short.pos) > len(long.pos) and short.read_length < long.read_length
    with api.Caller() as c:
        for w in (short, long, short):
            c.call(load(c, w))
            assert c.fetch().tobytes() == own_context(w)


def gap_workload(windows: int):
    """The reads of a small workload in the first window and again in the last,
    and in a window between them as reads of several hits, which leave no
    record: that one takes another's likelihood, and the empty ones show
    another's counts."""
    w = edge_workload("plain")
    n, G = w.config.genome_len, windows * 262144 + w.config.genome_len
    at = [0, windows // 2 * 262144 + 500, G - n]
    ref = np.frombuffer(b"ACTG", dtype=np.uint8)[np.random.default_rng(windows).integers(0, 4, G)]
    for x in at:
        ref[x:x + n] = w.ref
    thrice = lambda x: np.concatenate([x, x, x])
    return dataclasses.replace(w, ref=ref, config=dataclasses.replace(w.config, genome_len=G),
                               pos=np.concatenate([w.pos + x for x in at]).astype(np.int32), length=thrice(w.length),
                               hit=np.concatenate([w.hit, np.full_like(w.hit, 2), w.hit]), strand=thrice(w.strand),
                               seq=thrice(w.seq), qual=thrice(w.qual), mismatch=thrice(w.mismatch))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32_FIXUP])
def test_longer_chromosome_with_gap_windows(precision, native_lib):
    """Kept counts and likelihoods of a longer chromosome than those they were
    made for."""
    first, longer, plain = gap_workload(2), gap_workload(6), edge_workload("plain")
    with api.Caller() as c:
        for w in (plain, first, longer, plain, first):
            c.call(load(c, w, precision))
            got, text = c.fetch().tobytes(), c.format_cns("chr1")
            with api.Caller() as own:
                own.call(load(own, w, precision))
                assert got == own.fetch().tobytes()
                assert text == own.format_cns("chr1")


@pytest.mark.gpu
def test_recall_needs_a_resident_call_of_this_reference(native_lib):
    """Refused: before any call, after another reference, after only a streamed
    call, under another read length.  A streamed call in between leaves the
    resident alignments as they were."""
    w, other, long = edge_workload("plain"), gap_workload(2), edge_workload("lengths")
    refused = pytest.raises(RuntimeError, match=r"\(3\)")
    with api.Caller() as c:
        reads = load(c, w)
        with refused:
            c.recall_resident()
        c.call_streamed(reads)
        with refused:
            c.recall_resident()
        c.call(reads)
        want = c.fetch().tobytes()
        c.call_streamed(api.Caller.reads_struct(*[x[:300] for x in arrays(w)]))
        c.recall_resident()
        assert c.fetch().tobytes() == want
        # longer rows in the tables than on the device
        p = api.params_from_flags(long.config.flags, api.PRECISION_FP32_FIXUP)
        pm = c.calibrate(p, reads)
        c.load_tables(p, pm, c.prior_table(p), c.rank_table())
        with refused:
            c.recall_resident()
        with refused:
            c.tune(1)
        assert c.fetch().tobytes() == want
        reads = load(c, other)
        with refused:
            c.recall_resident()
        c.call(reads)
        want = c.fetch().tobytes()
        c.recall_resident()
        assert c.fetch().tobytes() == want


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32_FIXUP])
def test_recall_after_a_call_with_other_gap_windows(precision, native_lib):
    """A recall's graph holds the passes that the call's windows need: captured
    for alignments without gap windows, it is not replayed for as many with one."""
    gap = gap_workload(2)
    full = dataclasses.replace(gap, hit=np.ones_like(gap.hit))
    reads = {w: api.Caller.reads_struct(*a) for w, a in (("gap", arrays(gap)), ("full", arrays(full)))}
    with api.Caller() as c:
        load(c, gap, precision)
        for w in ("gap", "full"):
            c.call(reads[w])
        c.recall_resident()
        c.call(reads["gap"])
        p = api.params_from_flags(gap.config.flags + ["-e", "0.2"], precision)
        c.load_tables(p, c.calibrate(p, reads["gap"]), c.prior_table(p), c.rank_table())
        before = c.fetch().tobytes()
        c.recall_resident()
        got = c.fetch().tobytes()
        c.call(reads["gap"])
        assert got == c.fetch().tobytes() != before


@pytest.mark.gpu
def test_more_segments_than_any_call_before(native_lib, monkeypatch):
    """The control block grows in the middle of a call, between its uploads and
    its passes."""
    small, w = edge_workload("plain"), gap_workload(30)
    with api.Caller() as c:
        c.call(load(c, small))
        reads = load(c, w)
        monkeypatch.setenv("GSNP_SEGMENTS", "25")
        out = np.zeros(w.config.genome_len, dtype=api.SITE_DTYPE)
        c.call_into(reads, out.ctypes.data)
        monkeypatch.setenv("GSNP_SEGMENTS", "1")
        assert out.tobytes() == own_context(w)


@pytest.mark.gpu
def test_tables_that_cannot_be_made_change_nothing(native_lib):
    """A dependency coefficient above 1 is refused; the context goes on with the
    parameters and tables it has."""
    w, long = edge_workload("plain"), edge_workload("lengths")
    with api.Caller() as c:
        reads = load(c, w)
        c.call(reads)
        want = c.fetch().tobytes()
        p = api.params_from_flags(long.config.flags, api.PRECISION_FP64)
        pm = c.calibrate(p, reads)
        p.pcr_dependency = 0.1
        with pytest.raises(RuntimeError, match=r"\(2\).*dependency"):
            c.load_tables(p, pm, c.prior_table(p), c.rank_table())
        c.recall_resident()
        assert c.fetch().tobytes() == want
        c.call(reads)
        assert c.fetch().tobytes() == want


@pytest.mark.gpu
def test_reference_that_is_refused_changes_nothing(native_lib):
    """dbSNP rows that do not match the site codes, of a longer chromosome: the
    context keeps the reference and the calls it has."""
    w, longer = edge_workload("plain"), gap_workload(2)
    with api.Caller() as c:
        reads = load(c, w)
        c.call(reads)
        want, text = c.fetch().tobytes(), c.format_cns("chr1")
        codes = api.site_codes(longer.ref, np.array([7, 100000]))
        length = c.length
        rows = np.zeros(2, dtype=api.SNP_DTYPE)
        for pos in ((7,), (100000, 7), (7, 100001)):
            rows["pos"][:len(pos)] = pos
            with pytest.raises(RuntimeError, match=r"\(2\).*dbSNP"):
                c.load_reference(codes, rows[:len(pos)])
            c.length = length
            assert c.fetch().tobytes() == want and c.format_cns("chr1") == text
        c.recall_resident()
        assert c.fetch().tobytes() == want
        c.call(reads)
        assert c.fetch().tobytes() == want


@pytest.mark.gpu
def test_call_after_one_that_found_no_memory(native_lib):
    """Rows that no device holds (200 of 2 GB, never touched: no alignment has a
    base) end the call with an error; the next one allocates what it needs."""
    w = edge_workload("plain")
    with api.Caller() as c:
        reads = load(c, w)
        c.call(reads)
        want = c.fetch().tobytes()
        a = [x[:200].copy() for x in arrays(w)]
        a[1][:] = 0
        a[2][:] = 2
        huge = api.Caller.reads_struct(*a)
        huge.pitch = 2**31 - 1
        with pytest.raises(RuntimeError, match=r"\(1\).*memory"):
            c.call(huge)
        with pytest.raises(RuntimeError, match=r"\(1\).*memory"):
            c.call_streamed(huge)
        c.call(reads)
        assert c.fetch().tobytes() == want
        out = np.zeros(c.length, dtype=api.SITE_DTYPE)
        c.call_streamed(reads, None, out.ctypes.data)
        assert out.tobytes() == want
