"""A rule of csrc/core/launch.h that no run can show: kernels launched by launch_overlapped() are on the
SMs while their predecessor still writes what they will read, so they must not use loads that ask for
memory no kernel in flight writes (__ldg, ld.global.nc and the helpers built on it)."""

from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "csrc"
NON_COHERENT = re.compile(r"__ldg\s*\(|ld_input_v4\s*\(|\.global\.nc\b|Elem8<\w+>::load\([^;]*\bfalse\)"
                          r"|weighted_gather8<\w+>\([^;]*\bfalse\)")


def _code(path: Path) -> str:
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_overlapped_kernels_use_coherent_loads() -> None:
    launchers = [p for p in CSRC.rglob("*.cu") if "launch_overlapped(" in _code(p)]
    assert {"a2a_single.cu", "router.cu", "grouped_gemm.cu", "grouped_gemm_mx.cu"} <= {p.name for p in launchers}
    # router.cuh's and the GEMMs' headers hold device code of these kernels only
    for path in launchers + [CSRC / "ops" / h for h in ("router.cuh", "grouped_gemm_common.cuh", "tcgen05.cuh")]:
        found = NON_COHERENT.search(_code(path))
        assert found is None, f"{path.name}: {found.group(0)}"
