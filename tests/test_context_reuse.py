"""One context used for one chromosome after another, and with other tables in
between: what it keeps on the device has to fit each call, and the calls are
those of a context of their own."""
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
