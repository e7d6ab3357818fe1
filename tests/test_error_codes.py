"""A stage that gives up is seen by the call: every function of fire_api.cu that returns an error code is [[nodiscard]], and the
build refuses a source that drops such a code."""
import re
import subprocess

import pytest

from sparse_wf_gb300.build import CSRC, NVCC_FLAGS, nvcc


def test_error_codes_are_nodiscard():
    text = (CSRC / "fire_api.cu").read_text()
    found = re.findall(r"^(\[\[nodiscard\]\] )?cudaError_t (\w+)\(", text, re.M)
    assert len(found) > 15
    assert [name for mark, name in found if not mark] == []
    # a status is made from the codes: a refused contraction leaves no CUDA error behind
    for line in re.findall(r"!= cudaSuccess\)\s*\n?\s*return ([^;]*);", text):
        assert not line.startswith("launch_status"), line


@pytest.mark.parametrize("statement,builds", [("refused();", False), ("return refused();", True)])
def test_build_refuses_dropped_codes(tmp_path, statement, builds):
    src = tmp_path / "x.cu"
    src.write_text("#include <cuda_runtime.h>\n[[nodiscard]] cudaError_t refused() { return cudaErrorInvalidValue; }\n"
                   "cudaError_t stage() { %s return cudaSuccess; }\n" % statement)
    r = subprocess.run([nvcc(), *NVCC_FLAGS, "-c", str(src), "-o", str(tmp_path / "x.o")], capture_output=True, text=True)
    assert (r.returncode == 0) == builds, r.stderr
