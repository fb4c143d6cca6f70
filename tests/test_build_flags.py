"""The build keeps every a * b + c as two roundings, in device and in host code."""
import importlib.util
import os

from conftest import PKG


def test_no_contraction_on_either_side():
    spec = importlib.util.spec_from_file_location("mpp_build", os.path.join(PKG, "build.py"))
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    flags = build.flags()
    assert "-fmad=false" in flags
    assert "-ffp-contract=off" in flags[flags.index("-Xcompiler") + 1].split(",")
