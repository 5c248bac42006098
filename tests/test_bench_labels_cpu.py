"""The assembly kernels that bench.py names are ones the library launches."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LAUNCH = {"k_tile": "launch_tile", "k_rows": "launch_rows", "k_colored": "k_colored"}


def test_assembly_kernels_named_by_the_bench_exist():
    bench = open(os.path.join(ROOT, "bench.py")).read()
    impl = open(os.path.join(ROOT, "simit_gb300", "csrc", "sg_assemble_impl.cuh")).read()
    named = set(re.findall(r"\b(%s)<(\w+)>" % "|".join(LAUNCH), bench))
    assert named
    for kernel, elem in named:
        assert re.search(r"\b%s<%s\b" % (LAUNCH[kernel], elem), impl), (kernel, elem)
