import ctypes
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

# Tests that code or decode streams.  A library that was built without the
# reference's sources has stand-ins for its coders, which throw: these tests are
# then skipped with that reason, so that a run shows the others.
NEEDS_CODERS = {
    "test_cli_gpu.py": ["test_cli_archive", "test_cli_multiblock", "test_deferred_context_compresses_alike"],
    "test_learned_archive_gpu.py": ["test_learned_blocks_roundtrip_and_plain_mode_unchanged"],
    "test_learned_gpu.py": ["test_learned_coder_is_lossless_and_smaller"],
    "test_roundtrip_gpu.py": ["test_full_size_roundtrip"],
    "test_decode_cpu.py": ["test_cli_decompress", "test_corrupt_payloads_do_not_end_the_process", "test_decode_errors",
                           "test_decode_golden", "test_decode_multiblock", "test_decode_oracle_archive",
                           "test_decode_threads_agree", "test_python_wrapper", "test_random_small_archives"],
    "test_encode_cpu.py": ["test_block_body_matches_oracle", "test_missing_stream",
                           "test_random_block_bodies_match_oracle"],
    "test_oracle_golden.py": ["test_oracle_roundtrip_through_reference_decoder",
                              "test_oracle_writes_reference_archive_given_its_contested_links",
                              "test_unstable_reference_archive_is_pinned_up_to_its_mapping_tie"],
}


def built_without_coders():
    """Whether the library or the oracle has the stand-ins' failure (csrc/host/no_coders.hpp)."""
    for so in (("curc_b200", "libcurc_b200.so"), ("oracle", "_build", "liboracle.so")):
        path = os.path.join(ROOT, *so)
        if os.path.exists(path) and hasattr(ctypes.CDLL(path), "_ZN9no_coders4failEv"):
            return True
    return False


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and libcurc_b200.so")


def pytest_collection_modifyitems(items):
    mine = [i for i in items if getattr(i, "originalname", i.name) in NEEDS_CODERS.get(i.path.name, ())]
    if mine and built_without_coders():
        for i in mine:
            i.add_marker(pytest.mark.skip(reason="built without the reference's stream coders (its sources were absent)"))
