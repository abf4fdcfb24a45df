"""Test configuration: import paths for the package and the oracle, and the
`gpu` marker (tests that need a CUDA device; run with `-m gpu`)."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (os.path.join(ROOT, "ffr-pspw-dft-c_b200"), os.path.join(ROOT, "oracle"),
          os.path.join(ROOT, "tests")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); run with -m gpu")


# Tests that run the reference program itself (ref_program_case.py), which is
# built from its own sources by oracle/Makefile; where these are absent the tests
# have nothing to compare with.
REFERENCE_PROGRAM = {
    "test_scf_driver_gpu.py": {"test_cheby_scf_davidson_start_anderson",
                               "test_cheby_scf_random_start_pulay", "test_cheby_scf_kerker",
                               "test_cheby_scf_broyden", "test_cheby_scf_mixed_precision"},
    "test_system_gpu.py": {"test_device_setup_matches_reference"},
}


def pytest_collection_modifyitems(items):
    import pytest
    from ref_lib import ref_available
    if ref_available("libref.so"):
        return
    skip = pytest.mark.skip(reason="needs oracle/_ref/libref.so (the built reference)")
    for item in items:
        if getattr(item, "originalname", None) in REFERENCE_PROGRAM.get(item.path.name, ()):
            item.add_marker(skip)
