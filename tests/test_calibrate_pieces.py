"""The calibration pass over more alignments than its upload buffers hold at a
time, rows of odd lengths and a last piece of a few rows, against the matrix
computed with numpy from the same alignments; plain and packed."""
import numpy as np
import pytest

from gsnp_gb300 import api

CODE = np.full(256, 9, dtype=np.int64)
CODE[[65, 67, 84, 71]] = [0, 1, 2, 3]


def counts_of(ref, pos, length, hit, strand, seq, qual, qmin, qmax, L):
    """cpp/matrix.cc:58-118: [quality][cycle][reference][observed]"""
    nq = qmax - qmin + 1
    total = np.zeros(nq * L * 16, dtype=np.int64)
    cols = np.arange(seq.shape[1])[None, :]
    for i in range(0, pos.size, 20000):
        s = slice(i, i + 20000)
        ln, q, at = length[s][:, None], qual[s].astype(np.int64), pos[s][:, None].astype(np.int64)
        o = CODE[ref[np.minimum(at + cols, ref.size - 1)]]
        use = (cols < ln) & (hit[s] == 1)[:, None] & (at + ln < ref.size) & (o < 4) & (seq[s] != ord("N"))
        use &= (q >= qmin) & (q <= qmax)
        cyc = np.where((strand[s] != ord("+"))[:, None], ln - 1 - cols, cols)
        key = (((q - qmin) * L + cyc) * 4 + o) * 4 + ((seq[s] >> 1) & 3)
        total += np.bincount(key[use], minlength=total.size)
    return total.reshape(nq, L, 4, 4).astype(np.float64)


def matrix_of(n):
    """cpp/matrix.cc:129-205"""
    pm = np.ones(256 * 256 * 16)
    eye = np.eye(4, dtype=bool)
    for k in range(n.shape[0]):
        by = n[k].sum(axis=0)
        total, mism = by.sum(), by[~eye].sum()
        with np.errstate(invalid="ignore", divide="ignore"):
            cell = n[k] / n[k].sum(axis=2, keepdims=True)
            typ = by / by.sum(axis=1, keepdims=True)
        low = np.where(eye, (total - mism) / total, mism / total) if total > 0 else np.ones((4, 4))
        v = np.where(n[k] > 10, cell, np.where(by > 10, typ, low)[None])
        e = 10.0 ** (-(k / 10.0))
        v = np.where((v == 0) | (v == 1), np.where(eye, max(1 - e, 0.25), min(e / 3, 0.25)), v)
        for c in range(n.shape[1]):
            pm[(k << 12) | (c << 4):][:16] = v[c].ravel()
    return pm


@pytest.mark.gpu
@pytest.mark.parametrize("L,rows", [(255, 3 * ((32 << 20) // 255) + 3), (35, (32 << 20) // 35), (100, 17), (1, 1)])
def test_matrix_of_many_pieces(L, rows, native_lib):
    rng = np.random.default_rng(L)
    G = 100_003
    acgt = np.frombuffer(b"ACTGN", dtype=np.uint8)
    ref = acgt[rng.choice(5, G, p=[0.24, 0.25, 0.25, 0.25, 0.01])]
    pos = np.sort(rng.integers(0, G, rows)).astype(np.int32)
    length = rng.integers((L + 1) // 2, L + 1, rows).astype(np.int32)
    hit = np.where(rng.random(rows) < 0.1, 2, 1).astype(np.int32)
    strand = np.where(rng.random(rows) < 0.5, ord("-"), ord("+")).astype(np.uint8)
    cols = np.arange(L)[None, :]
    valid = cols < length[:, None]
    seq = ref[np.minimum(pos[:, None] + cols, G - 1)]
    odd = rng.integers(0, 256, seq.shape, dtype=np.uint8) < 4
    seq = np.where(odd, acgt[rng.integers(0, 5, seq.shape, dtype=np.uint8)], seq)
    qual = 66 + rng.integers(0, 38, seq.shape, dtype=np.uint8)
    seq, qual = np.where(valid, seq, 0).astype(np.uint8), np.where(valid, qual, 0).astype(np.uint8)
    p = api.params_from_flags(["-L", str(L), "-t", "-u"])
    want = matrix_of(counts_of(ref, pos, length, hit, strand, seq, qual, p.q_min, p.q_max, L))
    no_n = np.where(seq == ord("N"), ord("A"), seq).astype(np.uint8)   # a packed base is one of ACGT
    want_packed = matrix_of(counts_of(ref, pos, length, hit, strand, no_n, qual, p.q_min, p.q_max, L))
    packed = api.pack_reads(no_n, qual, length, p.q_min)
    plain = api.Caller.reads_struct(pos, length, hit, strand, seq, qual)
    small = api.Caller.reads_struct(pos, length, hit, strand, None, None, packed=packed, packed_qmin=p.q_min)
    with api.Caller() as c:
        c.load_reference(api.site_codes(ref))
        for reads, m in ((plain, want), (small, want_packed), (plain, want)):
            np.testing.assert_array_equal(c.calibrate(p, reads), m)
        if rows > 17:
            # refused as before, wherever the length is, and usable afterwards
            length[rows - 2] = L + 1
            with pytest.raises(RuntimeError, match="alignment %d is longer" % (rows - 2)):
                c.calibrate(p, plain)
            length[rows - 2] = L
            seq[rows - 2], qual[rows - 2] = ord("A"), 70
            want = matrix_of(counts_of(ref, pos, length, hit, strand, seq, qual, p.q_min, p.q_max, L))
            np.testing.assert_array_equal(c.calibrate(p, plain), want)
