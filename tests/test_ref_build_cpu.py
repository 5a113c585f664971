"""Without the reference tree, or with an empty folder in its place, building its
kernels is skipped and the prebuilt libraries, if any, are used."""
import os
import sys

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "oracle"))
import ref_frame  # noqa: E402


def test_no_reference_tree_builds_nothing(tmp_path):
    assert ref_frame.build(str(tmp_path)) == ref_frame.available()
    assert ref_frame.build(str(tmp_path / "missing")) == ref_frame.available()
