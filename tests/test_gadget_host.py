"""The one-call key switch and external product (abi_mlwe.cu) on a fake engine, without a
GPU: the route they take and what they do when the fake fails a call."""

from __future__ import annotations

import os
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def calls(tmp_path_factory):
    from vfhe_b200.build import ARCH, nvcc

    exe = tmp_path_factory.mktemp("gadget") / "gadget_host"
    # the entry points that the cases do not reach keep their symbols unresolved
    subprocess.run([nvcc(), *ARCH, "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-Xlinker",
                    "--unresolved-symbols=ignore-all", "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "gadget_host.cu"), "-o", str(exe)], check=True)

    def run(entry: str, case: str) -> dict[str, int]:
        r = subprocess.run([str(exe), entry, case], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), check=True,
                           capture_output=True, text=True, timeout=60)
        return {k: int(n) for k, n in (line.split() for line in r.stdout.splitlines())}

    return run


@pytest.mark.parametrize("entry", ["keyswitch", "external_product"])
@pytest.mark.parametrize("case", ["transform_fails", "launch_fails", "no_scratch"])
def test_a_failed_product_gives_its_scratch_back_and_stops(calls, entry, case):
    """The output is neither divided nor added to; its extended rows are zeroed instead of left
    as they were."""
    got = calls(entry, case)
    assert got["error"] >= 1
    assert got.get("alloc", 0) == got.get("free", 0) == (0 if case == "no_scratch" else 1)
    assert "divide" not in got and "add" not in got
    assert got["zero"] == 1


@pytest.mark.parametrize("entry", ["keyswitch", "external_product"])
def test_a_large_digit_outside_the_key_goes_digit_by_digit(calls, entry):
    got = calls(entry, "large_digit")
    assert "alloc" not in got and got["product"] >= 6


@pytest.mark.parametrize("entry,case", [
    ("keyswitch", "key_mask_is_output_body"), ("keyswitch", "key_body_is_output_mask"),
    ("keyswitch", "output_mask_is_output_body"), ("keyswitch", "input_mask_is_output_body"),
    ("external_product", "key_mask_is_output_body"), ("external_product", "key_body_is_output_mask"),
    ("external_product", "output_mask_is_output_body"), ("external_product", "input_mask_is_output_body"),
    ("external_product", "input_body_is_output_mask"), ("external_product", "input_body_is_output_body")])
def test_shared_polynomials_go_digit_by_digit(calls, entry, case):
    """The output is zeroed before an input is read, and the product whose operands share a
    polynomial (3 digits, 2 components) is taken one digit and component after the other."""
    got = calls(entry, case)
    assert got["zero"] == 1 and got["product"] >= 6


@pytest.mark.parametrize("entry", ["keyswitch", "external_product"])
@pytest.mark.parametrize("case", ["key_rows_moved", "output_rows_moved", "digit_rows_moved"])
def test_rows_out_of_order_go_digit_by_digit(calls, entry, case):
    """A polynomial's rows are where its row pointers say; the block's order is not assumed."""
    assert calls(entry, case)["product"] >= 6


@pytest.mark.parametrize("entry", ["keyswitch", "external_product"])
def test_separate_polynomials_take_every_digit_at_once(calls, entry):
    got = calls(entry, "plain")
    assert got["alloc"] == got["free"] == (1 if entry == "keyswitch" else 2)
    assert "product" not in got and "error" not in got and got["divide"] == 1
