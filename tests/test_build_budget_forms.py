"""Register budget, from the build's `-Xptxas -v` reports as in test_build_budget.py, of the Hermite forms that
its patterns leave out: the j-paired forms over j-lanes and with the best j-quad, and the integrator's step
kernel."""
import re

import pytest

from test_build_budget import ptxas_report

# g6_kernel<128, 2, JL, double-float positions, NN, no lists, JP>: every j-paired form of 128 threads
JPAIRED = re.compile(r"_ZN3pgb9g6_kernelILi128ELi2ELi([12])ELb1ELb[01]ELb0ELi([123])EEEv")
# hm_run_kernel<double-float positions, START>
STEP = re.compile(r"_ZN3pgb13hm_run_kernelILb([01])ELb([01])EEEv")


@pytest.mark.parametrize("lib", ["libpg6", "libpg6_newton"])
def test_every_j_paired_form(lib):
    hits = {k: v for k, v in ptxas_report(lib).items() if JPAIRED.match(k)}
    assert {JPAIRED.match(k).groups() for k in hits} == {("1", "1"), ("1", "2"), ("1", "3"), ("2", "3")}
    for k, (regs, spill) in hits.items():
        assert spill == 0, f"{lib} {k}: {spill} bytes of spill stores"
        assert regs <= 168, f"{lib} {k}: {regs} registers, above the 3-CTA budget"


@pytest.mark.parametrize("lib", ["libpg6", "libpg6_newton"])
def test_step_kernel(lib):
    """Two CTAs of 256 threads an SM: 128 registers.  The start-up instance spills nothing; the one of the
    block steps does with its small steps' four task shapes (620 bytes over all of them, 40 without: the
    bound is that and two doubles a shape)."""
    hits = {STEP.match(k).groups(): v for k, v in ptxas_report(lib).items() if STEP.match(k)}
    assert set(hits) == {(a, b) for a in "01" for b in "01"}
    for (_, start), (regs, spill) in hits.items():
        assert regs <= 128
        assert spill <= (0 if start == "1" else 684)
