"""Calls that need no set-up of the device run without one."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def decode(pkg, n_in, n_out):
    """The dense decode through the bare entry point, no qtip_init before it."""
    gen = torch.Generator().manual_seed(n_in)
    trellis = torch.randint(-32768, 32768, (n_in * n_out // 256 * 32,), generator=gen, dtype=torch.int16).cuda()
    lut = torch.randint(-2 ** 31, 2 ** 31, (1024,), generator=gen).to(torch.int32).cuda()
    out = torch.zeros(n_out, n_in, dtype=torch.int16, device="cuda")
    m = pkg._lib.QtipMatrix(trellis.data_ptr(), None, None, lut.data_ptr(), n_in, n_out)
    pkg.lib().call("qtip_decode_matrix", m, C.c_void_p(out.data_ptr()), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return out.cpu()


SHAPES = ((384, 64), (256, 32 * 500), (1024, 16384))


def test_dense_decode_needs_no_init(gpu, tmp_path):
    out = str(tmp_path / "out.pt")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], cwd=ROOT, check=True, timeout=300)
    for shape, got in zip(SHAPES, torch.load(out)):
        assert torch.equal(got, decode(gpu, *shape)), shape


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    import __graft_entry__
    package = __graft_entry__.load_package()
    torch.save([decode(package, *s) for s in SHAPES], sys.argv[1])
