"""Kernels launched programmatically run beside the launch that writes their inputs until pdl_wait: what that
launch wrote is read with plain loads (ld_dep, ld_after); read-only loads (__ldg) are for the neighbour table alone."""
import re
from pathlib import Path

import pytest

DEVICE = Path(__file__).resolve().parents[1] / "dg_b200" / "csrc" / "device"


@pytest.mark.parametrize("header,name", [
    ("kernels.cuh", "res1d_load"), ("kernels.cuh", "res_lim1d_chain_kernel"), ("kernels.cuh", "wavespeed_kernel"),
    ("limiter2d_tile.cuh", None), ("tile2d_cols.cuh", None), ("tile2d_ordered.cuh", None)])
def test_no_read_only_loads_of_state(header, name):
    text = (DEVICE / header).read_text()
    if name:  # one function: from its name to the closing brace of the file's indentation
        text = text[text.index(name + "("):]
        text = text[:text.index("\n}\n")]
    assert "ld_dep(" in text or "ld_after(" in text
    assert [a for a in re.findall(r"__ldg\(([\w.]+)", text) if a not in ("nbr", "a.nbr")] == []
    assert re.findall(r"(?:if \(|[=:?&|] )(?:a\.)?scal->(?:flags|dt)\b", text) == []
