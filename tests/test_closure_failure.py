"""A closure whose network cannot be enqueued fails the step. The failure is made on the host: where there is no driver its
tensor maps cannot be made, before anything is launched, and the step's own launches would report another error."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include "gam_closure.cu"
int main() {
    gam_closure C;
    gam::Handle h;
    C.L = h.L = make_lay(8, 8, 8);
    C.box.P = C.L.P; C.box.Q = C.L.Q; C.box.E = C.L.E;
    C.box.c0 = (long long)C.L.P * C.L.Q + C.L.P + 1;
    C.box.c1 = C.L.E - C.box.c0;
    h.p.doMHD = 1;
    h.closure = &C;
    for (int part : {gam::STEP_ALL, gam::STEP_POST}) std::printf("%d\\n", gam::step_enqueue(h, 0, nullptr, false, part));
    std::printf("%d\\n", gam::net_init());
    return 0;
}
"""


def test_step_reports_a_network_that_cannot_be_enqueued(tmp_path):
    import torch
    if torch.cuda.is_available():
        pytest.skip("the tensor maps can be made here")
    from kaiju_b200 import build as kb
    kb.build()
    src, exe = tmp_path / "step.cu", tmp_path / "step"
    src.write_text(SRC)
    subprocess.run([kb.NVCC, *kb.ARCH, "-std=c++17", "-I", kb.CSRC, "-I", os.path.join(ROOT, "include"), str(src), "-o",
                    str(exe), "-L", kb.HERE, "-lgamgpu", "-Xlinker", "-rpath," + kb.HERE], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    invalid_value, not_supported = "1", "801"   # cudaErrorInvalidValue, cudaErrorNotSupported
    assert out == [invalid_value, invalid_value, not_supported]
