"""The cns text at the edges of its blocks (128 rows) and pieces (262,144
rows): genomes that end on, before and after them, chromosome names of every
alignment and of the longest length, buffers shorter than the text, and the
file writer, against the CPU oracle's text, byte for byte."""
import ctypes

import numpy as np
import pytest

from gsnp_gb300 import api, synth

from oracle_run import flags_for, oracle_outputs


def format_into(c, name: str, buf: np.ndarray, cap: int) -> int:
    size = ctypes.c_int64(cap)
    assert c.lib.gsnp_format_cns(c.ctx, name.encode(), buf.ctypes.data, ctypes.byref(size)) == 0
    return size.value


@pytest.mark.gpu
@pytest.mark.parametrize("sites", [20095, 20096, 20097, 262144, 3 * 262144 + 77])
def test_text_at_block_and_piece_edges(sites, tmp_path, oracle_bin, native_lib):
    w = synth.make_workload("c0", genome_len=sites)
    paths = synth.write_inputs(w, str(tmp_path))
    flags = flags_for(w, paths)
    ref = oracle_outputs(oracle_bin, w, flags, str(tmp_path))
    assert ref["rc"] == 0, ref["stderr"]
    want = ref["cns"]
    old = w.chr_name.encode() + b"\t"
    rows = want.split(b"\n")[:-1]
    assert len(rows) == sites and all(r.startswith(old) for r in rows)
    c, _, _ = api.run_workload(w, flags)
    try:
        assert c.format_cns(w.chr_name) == want
        for name in ["x", "chromosome_12_B", "n" * 254, "n" * 255]:
            new = name.encode() + b"\t"
            text = b"".join(new + r[len(old):] + b"\n" for r in rows)
            assert c.format_cns(name) == text
        # a shorter buffer gets the first bytes, and nothing after them is touched
        for cap in [0, 1, 15, len(want) // 2 + 3, len(want) - 1, len(want)]:
            buf = np.full(len(want) + 64, 0xEE, dtype=np.uint8)
            assert format_into(c, w.chr_name, buf, cap) == cap
            assert buf[:cap].tobytes() == want[:cap] and (buf[cap:] == 0xEE).all()
        path = tmp_path / "out.cns"
        assert c.lib.gsnp_write_cns(c.ctx, w.chr_name.encode(), str(path).encode()) == 0
        assert path.read_bytes() == want
        with pytest.raises(Exception):
            c.format_cns("n" * 256)
    finally:
        c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("streamed", [False, True])
def test_value_outside_the_formatter_is_an_error(streamed, tmp_path, native_lib):
    """A rank-sum value that the exact formatter cannot print, in the first of
    two chunks only, ends the text with an error however it is written."""
    import dataclasses
    from test_lean import edge_workload
    w = edge_workload("plain")
    ref = np.concatenate([w.ref, np.full(262144, ord("A"), dtype=np.uint8)])
    w = dataclasses.replace(w, ref=ref, config=dataclasses.replace(w.config, genome_len=ref.size))
    c, reads, pm = api.run_workload(w, list(w.config.flags))
    try:
        assert len(c.format_cns("chr1")) > 0
        p = api.params_from_flags(w.config.flags)
        c.load_tables(p, pm, c.prior_table(p), np.full(64 * 64 * 2048, 1e-30))
        with pytest.raises(RuntimeError, match=r"\(3\).*formatter"):
            if streamed:
                c.set_option("stream_windows", 1)
                c.call_streamed(reads, "chr1", None, str(tmp_path / "cns"))
            else:
                c.call(reads)
                c.format_cns("chr1")
    finally:
        c.close()
