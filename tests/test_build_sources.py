"""What goes into the library (cmaq_gb300/build.py)."""
import re

from cmaq_gb300 import build as b


def test_no_tables_that_no_kernel_reads():
    kernels = [p for p in b.CSRC.glob("*.cu*")]
    assert kernels and not [p.name for p in kernels if re.search(r"\bM::gw_|\bGW_N", p.read_text())]
    names = [p.name for p in b.sources()]
    assert not [n for n in names if "gw_tables" in n]
    assert {"chem_capi.cu", "kmt2.cu", "cb6r5_ae7_aq_coop.cu", "cracmm2_coop.cu", "cracmm2_rates.cu"} <= set(names)
