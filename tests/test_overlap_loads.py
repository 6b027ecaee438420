"""Kernels launched with launch_dependent are resident while the kernel before them still writes: they may use read-only loads
(__ldg, or parameters that are pointers to const with __restrict__) only for data no kernel of the chain writes."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mxmoe_b200" / "csrc"
FILES = sorted(p.name for p in CSRC.glob("*.cu") if '#include "launch.cuh"' in p.read_text())
# weight scales (and zero points), sign vectors, Hadamard factors, problem lists
CONSTANT = re.compile(r"scale_b|szp|signs|hadK|problems")


def _calls(text: str, name: str):
    """The argument of every call of `name`, parentheses matched."""
    for m in re.finditer(re.escape(name) + r"\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        yield text[m.end():i - 1]


def test_files_are_found():
    assert {"act_kernels.cu", "route_kernels.cu", "had_kernels.cu", "gg_duo_kernel.cu", "gg_swap_kernel.cu"} <= set(FILES)


@pytest.mark.parametrize("name", FILES)
def test_read_only_loads_take_constant_data(name):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    assert [a for a in _calls(text, "__ldg") if not CONSTANT.search(a)] == []
    assert [p for p in re.findall(r"const [\w:]+\s*\* __restrict__ \w+", text) if not CONSTANT.search(p)] == []
    assert "ld.global.nc" not in text


@pytest.mark.parametrize("name", FILES)
def test_waits_come_before_the_first_access(name):
    """Every kernel (or the body it calls first) starts with the wait; the grouped GEMMs set up barriers and tensor memory first."""
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    if name.startswith("gg_"):
        head = text[:text.index("grid_dependency_wait();   " if "grid_dependency_wait();   " in text else "build_sched(sc")]
        body = head[head.index("extern __shared__"):]
        assert "problems[" not in body and "build_sched" not in body
        assert set(re.findall(r"status->(\w+)", body)) <= {"error", "timeout_ms"}
        return
    bodies = re.findall(r"__global__ void[^{;]*\{\s*([^\n]*)\n\s*([^\n]*)", text)
    bodies = [b for b in bodies if "rows_quant_body<" not in b[0]] + \
        re.findall(r"void rows_quant_body\([^{;]*\{\s*([^\n]*)\n\s*([^\n]*)", text)
    assert bodies
    for first, second in bodies:
        assert first.startswith("release_dependents();") and second.startswith("grid_dependency_wait();")


def test_only_single_block_launches_release_early():
    """Launches of several blocks that released early made the step behind them slower (61 tokens mixed by 3 %)."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "launch.cuh").read_text())
    assert re.search(r"if \(gridDim\.x == 1\) asm volatile\(\"griddepcontrol\.launch_dependents;\"", text)
    assert sum(p.read_text().count("griddepcontrol.launch_dependents") for p in CSRC.iterdir()) == 1


@pytest.mark.gpu
@pytest.mark.skipif(shutil.which("nvcc") is None, reason="no nvcc")
def test_a_refused_launch_is_reported_once(tmp_path):
    """launch_dependent returns the error and leaves none behind for the next check of the runtime's last error (a block of 4096
    threads is refused on the host)."""
    (tmp_path / "t.cu").write_text('''
#include "launch.cuh"
__global__ void k(int) {}
int main() {
  const cudaError_t e = mxb::launch_dependent(k, 1, 4096, 0, (cudaStream_t)0, 0);
  return (e != cudaSuccess && cudaPeekAtLastError() == cudaSuccess) ? 0 : 1;
}
''')
    exe = tmp_path / "t"
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-I", str(CSRC), "-o", str(exe),
                    str(tmp_path / "t.cu")], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
