"""The autotuner's report (gsnp_tune)."""
import re

import pytest

from gsnp_gb300 import api, synth


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [api.PRECISION_FP64, api.PRECISION_FP32_FIXUP])
def test_summary_has_the_fastest_of_each_path(precision, native_lib):
    """The times that decide between the two paths are those of the best binned
    and the best persistent measurement, in either form."""
    w = synth.make_workload("c1", scale=0.02)
    c, _, _ = api.run_workload(w, [f for f in w.cli_flags("dbsnp") if f != "-C"], precision=precision)
    try:
        report = c.tune(2)
    finally:
        c.close()
    binned = [float(x) for x in re.findall(r"^binned limits .*: ([\d.]+) ms$", report, re.M)]
    persistent = [float(x) for x in re.findall(r"^persistent slots .*: ([\d.]+) ms$", report, re.M)]
    summary = re.search(r"^# sample: .* best binned ([\d.]+) ms, best persistent ([\d.]+) ms$", report, re.M)
    assert (float(summary[1]), float(summary[2])) == (min(binned), min(persistent)), report
    if min(binned) != min(persistent):
        assert re.search(r"^persistent (\d)$", report, re.M)[1] == str(int(min(persistent) < min(binned)))
