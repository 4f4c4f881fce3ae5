"""What the tcgen05 kernels' sources have to keep and no run can show for certain, and their host side (no GPU)."""

import re
import subprocess
import sys
from pathlib import Path

import pytest

import ondeviceinfer_b200

CSRC = Path(ondeviceinfer_b200.__file__).parent / "csrc"


def _code(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def test_no_load_from_tensor_memory_is_left_on_its_way():
    """tcgen05.ld writes its registers when it likes until the wait that names them.  The grouped product's epilogue asks for 16 columns ahead:
    it may ask for no more of them than its loop goes through and waits for, and the loop may not be left in between."""
    text = _code("grouped_tcgen05.cu")
    loop = re.search(r"for \(int c = 0; c < (\w+); c \+= 16\) \{(.*?)tc_fence_before\(\)", text, re.S)
    bound, body = loop.group(1), loop.group(2)
    loads = re.findall(r"^(.*)tmem_ld16\(src", text, re.M)
    assert [load.strip() for load in loads] == [f"if ({bound} > 0)", f"if (c + 16 < {bound})"]
    assert "break" not in body and body.index("tmem_wait16(next)") < body.index("tmem_ld16(")


ISSUING = [p.name for p in sorted(CSRC.glob("*.cu")) if "elect_one()" in _code(p.name)]


@pytest.mark.parametrize("name", ISSUING)
def test_a_warp_that_issues_waits_as_one(name):
    """The warps that issue MMAs go through their loops whole, and the lane that issues waits for nobody: every wait there has to rejoin the
    warp (``warp_wait``), or a lane a lap of the ring behind waits for a phase that is over and, two seconds later, ends the block."""
    text = _code(name)
    at = text.index("elect_one()")
    branch = text[at:text.index("} else ", text.index("umma_commit", at))]
    assert "warp_wait(" in branch and "mbar_wait(" not in branch


def test_the_kernels_that_issue_are_all_here():
    assert ISSUING == ["attention_tcgen05.cu", "gemm_f32_split.cu", "gemm_prefill_tcgen05.cu", "gemm_tcgen05.cu", "grouped_tcgen05.cu"]


@pytest.mark.parametrize("name", ["gemm_f32_split.cu", "grouped_tcgen05.cu"])
def test_shared_memory_is_asked_for_on_every_device(name):
    """The limit of a kernel's shared memory is the device's: a thread that goes on to another one has to set it there too."""
    text = _code(name)
    assert text.count("cudaFuncSetAttribute(") == 1
    condition = re.findall(r"if \(([^{]*)\) \{", text[:text.index("cudaFuncSetAttribute(")])[-1]
    assert re.search(r"\bdevice != \w+", condition) and "cudaGetDevice(" in text


def test_a_product_without_rows_needs_no_scratch():
    """The plan divides by the tiles of rows: a call without any has to come back, not end the process."""
    script = ("from ctypes import c_long\n"
              "from ondeviceinfer_b200.kernels.build import load_library\n"
              "lib = load_library('gemm_f32_split')\n"
              "lib.odi_gemm_f32_split_scratch.restype = c_long\n"
              "print([lib.odi_gemm_f32_split_scratch(*s) for s in ((0, 2048, 2048), (3, 0, 2048), (3, 2048, 0), (-1, 2048, 2048))])\n")
    done = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, cwd=CSRC.parents[1])
    assert done.returncode == 0 and done.stdout.strip() == "[0, 0, 0, 0]", (done.returncode, done.stderr)


def test_the_chunks_of_the_delta_rules_scan_begin_where_shared_memory_does():
    """Static shared variables come first: 16 bytes of them put every row of the chunks across one more 128-byte line, 4 to 9 % of the mixer."""
    text = _code("delta_chunk.cuh")
    kernel = text[text.index("dc_scan_kernel(DeltaChunkArgs a)"):text.index("static int dc_launch_form")]
    assert [line for line in kernel.splitlines() if "__shared__" in line] == ["  extern __shared__ __align__(16) float dc_smem[];"]
