"""FP32 attention of short sequences at every length it is served at.  How much shared
memory a launch takes grows with the length, and from 48 KiB on the kernel's limit has to
be raised first: it stays raised for the lengths after it, so each head width runs in a
process of its own, shortest first."""
import glob
import os
import re
import subprocess
import sys

import pytest

from conftest import PACKAGE, REPO

LENGTHS = 128


def test_every_byte_of_a_launch_is_counted():
    """The launch sites that raise a limit from 48 KiB on look at dynamic bytes: their
    kernels have no others."""
    counting = [path for path in glob.glob(os.path.join(PACKAGE, "csrc", "attention*.cu"))
                if re.search(r"bytes > 48 \* 1024", open(path).read())]
    assert len(counting) == 3, counting
    for path in counting:
        with open(path) as source:
            for line in source:
                code = line.split("//")[0]
                assert "__shared__" not in code or "extern __shared__" in code, (path, line)


@pytest.mark.gpu
@pytest.mark.parametrize("head_dim", [8, 16, 32, 64])
def test_every_length(head_dim):
    """Largest error against the largest entry, in 64 bits: 1e-5 forward, 2e-5 backward
    (sums of up to 128 terms, 6e-8 each, behind exponentials of 2e-7)."""
    done = subprocess.run([sys.executable, os.path.abspath(__file__), str(head_dim)],
                          stdout=subprocess.PIPE, timeout=600, cwd=REPO)
    found = re.findall(r"^length (\d+) (\S+) (\S+)$", done.stdout.decode(), re.M)
    assert done.returncode == 0 and len(found) == LENGTHS, (found[-1:], done.stdout[-500:])
    for length, forward, backward in found:
        assert float(forward) <= 1e-5 and float(backward) <= 2e-5, (length, forward, backward)


def main(head_dim):
    import ctypes
    import numpy as np
    import torch
    from oracle import vit_oracle as vo
    lib = ctypes.CDLL(os.path.join(PACKAGE, "libvitb200.so"))
    groups, scale = 3, 1.0 / np.sqrt(head_dim)
    for length in range(1, LENGTHS + 1):
        rng = np.random.RandomState(length)
        rows = groups * length
        q, k, v, dout = (rng.randn(rows, head_dim).astype(np.float32) for _ in range(4))
        inputs = [torch.from_numpy(x).cuda() for x in (q, k, v)]
        upstream, out = torch.from_numpy(dout).cuda(), torch.empty(rows, head_dim).cuda()
        grads = [torch.zeros(rows, head_dim).cuda() for _ in range(3)]

        def pointers(*tensors):
            return [ctypes.c_void_p(t.data_ptr()) for t in tensors]

        sizes = (ctypes.c_size_t(groups), ctypes.c_size_t(length), ctypes.c_size_t(head_dim),
                 ctypes.c_float(scale), 1, None)
        assert lib.vitb200_k_attention(*pointers(*inputs), None, *pointers(out),
                                       *sizes) == 0, length
        assert lib.vitb200_k_attention_backward(
            *pointers(*inputs), None, *pointers(out, upstream, *grads), None,
            *sizes) == 0, length
        torch.cuda.synchronize()
        q, k, v, dout = (x.astype(np.float64) for x in (q, k, v, dout))
        p, want = vo.multi_head_attention(q, k, v, groups, length, scale)
        slopes = vo.multi_head_attention_backward(q, k, v, p, dout, groups, length, scale)

        def worst(got, expected):
            return float(np.abs(got.cpu().numpy() - expected).max() / np.abs(expected).max())

        # (One key: its probability is one whatever the scores, so that what is left of
        # their gradients is rounding.)
        kept = (0, 1, 2) if length > 1 else (2,)
        print("length", length, worst(out, want),
              max(worst(grads[i], slopes[i]) for i in kept), flush=True)


if __name__ == "__main__":
    sys.path.insert(0, REPO)
    main(int(sys.argv[1]))
