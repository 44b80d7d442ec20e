"""The rule that lets the gradient kernels write a caller's buffer in place
(csrc/host/direct_output.h), compiled and run on the CPU: memory of the
context's own device, 16-byte aligned, apart from the records; and the
gradients through buffers on either side of it."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from atlas_rt import build as atlas_build

REPO = Path(__file__).resolve().parent.parent

PROGRAM = r"""
#include "direct_output.h"
#include <cstdio>
using atlas::rt::host::DirectOutput;
int main() {
    auto at = [](unsigned long long v) { return reinterpret_cast<const void*>(v); };
    const cudaMemoryType types[] = { cudaMemoryTypeUnregistered, cudaMemoryTypeHost, cudaMemoryTypeDevice,
                                     cudaMemoryTypeManaged };
    for (cudaMemoryType t : types)
        for (int dev = 0; dev < 2; dev++) {
            cudaPointerAttributes a{};
            a.type = t;
            a.device = dev;
            std::printf("%d %d %d\n", int(t), dev, int(DirectOutput(a, 1, at(0x10000), 4096, at(0x90000), 640)));
        }
    cudaPointerAttributes a{};
    a.type = cudaMemoryTypeDevice;
    a.device = 1;
    // aligned to 8 and 4 bytes, null; records right behind, right before, and over either end of it
    const unsigned long long out[] = { 0x10008, 0x10004, 0, 0x10000, 0x10000, 0x10000, 0x10000, 0x10000 };
    const unsigned long long in[] = { 0x90000, 0x90000, 0x90000, 0x11000, 0xfd80, 0x10ff0, 0xfd90, 0x10100 };
    for (int i = 0; i < 8; i++) std::printf("%d\n", int(DirectOutput(a, 1, at(out[i]), 4096, at(in[i]), 640)));
}
"""


def test_rule(tmp_path):
    cuda = Path(atlas_build._cuda_lib_dir(atlas_build._nvcc())).parent
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", f"-I{atlas_build.CSRC / 'host'}",
                        f"-I{cuda / 'include'}", str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lines = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split("\n")
    # unregistered 0, host 1, device 2, managed 3 on devices 0 and 1, for a context of device 1
    assert lines[:8] == [f"{t} {d} {int((t, d) == (2, 1))}" for t in range(4) for d in range(2)]
    assert lines[8:16] == ["0", "0", "0", "1", "1", "0", "0", "0"]


@pytest.mark.gpu
def test_gradients_into_either_kind_of_buffer():
    """Device buffers take them directly, managed memory and a buffer that the
    records lie in through the cache's own: the same gradients."""
    import torch
    import atlas_rt
    from test_rc_gpu import HI, LO, random_records, rel
    rt = C.CDLL(str(next(Path(atlas_build._cuda_lib_dir(atlas_build._nvcc())).glob("libcudart.so*"))))
    ctx = atlas_rt.Context(device=0)
    rc = atlas_rt.RadianceCache(ctx, LO, HI, log2_table=14, seed=3)
    managed = C.c_void_p()
    try:
        rec = random_records(700, 9)
        q = torch.from_numpy(rec).cuda()
        want = [torch.zeros(k, device="cuda") for k in (rc.n_mlp, rc.n_grid)]
        loss = rc.gradients(q, *want)
        want = [w.cpu().numpy() for w in want]
        # the records at the front of the buffer that the grid's gradients go to
        both = torch.zeros(rc.n_grid, device="cuda")
        both[:rec.size] = q.reshape(-1)
        assert both.data_ptr() % 16 == 0 and rec.size < rc.n_grid
        mlp = torch.zeros(rc.n_mlp, device="cuda")
        assert np.isclose(rc.gradients(both[:rec.size].view(-1, 16), mlp, both), loss, rtol=1e-5)
        assert rel(mlp.cpu().numpy(), want[0]) < 1e-5 and rel(both.cpu().numpy(), want[1]) < 1e-5
        assert rt.cudaMallocManaged(C.byref(managed), C.c_size_t(4 * rc.n_mlp), 1) == 0
        view = np.ctypeslib.as_array(C.cast(managed, C.POINTER(C.c_float)), (rc.n_mlp,))
        view[:] = 3.0
        got = np.zeros(rc.n_grid, np.float32)
        assert np.isclose(rc.gradients(q, view, got), loss, rtol=1e-5)
        assert rel(np.array(view), want[0]) < 1e-5 and rel(got, want[1]) < 1e-5
    finally:
        torch.cuda.synchronize()
        if managed:
            rt.cudaFree(managed)
        rc.close()
        ctx.close()
