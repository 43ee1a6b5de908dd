"""A product whose first call in a process is captured into a graph: nothing that it sets
up may end the capture (FP32 FMAs need nothing; the tensor-core kernels a word of mapped
memory for their status)."""
import os
import re
import subprocess
import sys

import pytest

from conftest import PACKAGE, REPO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,bound", [(1, 4e-7), (2, 1e-3)], ids=["fp32", "tf32"])
@pytest.mark.parametrize("rows", [500, 12800])
def test_first_call_is_captured(rows, precision, bound):
    """2-norm against 64 bits: FP32 sums of up to 384 terms as FMAs take them, TF32 operands
    of 10 bits."""
    done = subprocess.run([sys.executable, os.path.abspath(__file__), str(rows),
                           str(precision)], stdout=subprocess.PIPE, timeout=300, cwd=REPO)
    found = re.findall(r"^error (\S+)$", done.stdout.decode(), re.M)
    assert done.returncode == 0 and len(found) == 3, done.stdout.decode()[-500:]
    assert all(float(error) <= bound for error in found), found


def main(m, precision):
    import ctypes
    import torch
    lib = ctypes.CDLL(os.path.join(PACKAGE, "libvitb200.so"))
    k, n = 128, 384
    x, w, dy = (torch.randn(*shape, device="cuda") for shape in ((m, k), (k, n), (m, n)))
    y, dx, dw = (torch.zeros(*shape, device="cuda") for shape in ((m, n), (m, k), (k, n)))
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def pointers(*tensors):
        return [ctypes.c_void_p(t.data_ptr()) for t in tensors]

    with torch.cuda.graph(graph, stream=stream):
        sizes = (*(ctypes.c_size_t(s) for s in (m, k, n)), precision,
                 ctypes.c_void_p(stream.cuda_stream))
        assert lib.vitb200_k_gemm(*pointers(x, w, y), *sizes) == 0
        assert lib.vitb200_k_gemm_backward(*pointers(x, w, dy, dx, dw), *sizes) == 0
    graph.replay()
    torch.cuda.synchronize()
    x, w, dy = x.double(), w.double(), dy.double()
    for got, want in ((y, x @ w), (dx, dy @ w.T), (dw, x.T @ dy)):
        print("error", float((got.double() - want).norm() / want.norm()), flush=True)


if __name__ == "__main__":
    main(int(sys.argv[1]), int(sys.argv[2]))
