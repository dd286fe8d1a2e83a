"""Chained launches (programmatic dependent launch) against plain stream order: the same calls on the same buffers, again and
again, give the same bits. The plain side runs in a process of its own with QTIP_PDL=0."""
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
STEPS = 24


def decode_steps(gpu, tokens, n_in=1536, n_out=1792):
    """STEPS times prepare -> codes of this step into the matrix -> product -> finish, with nothing between the launches: the
    product directly follows the kernel that writes its codes, and one step writes what the one before still reads."""
    lin, gen = gpu.linear, torch.Generator(device="cuda").manual_seed(tokens)
    packed = torch.randint(-32768, 32768, (2, (n_out // 16) * (n_in // 16), 32), generator=gen, device="cuda", dtype=torch.int16)
    su, sv = (torch.randint(0, 2, (n,), generator=gen, device="cuda").float() * 2 - 1 for n in (n_in, n_out))
    w = lin.Matrix(torch.zeros(packed[0].numel(), dtype=torch.int16, device="cuda"), su, sv,
                   lin.runtime_lut(gpu.synth.seeded_tlut(1)), n_in, n_out)
    x = torch.randn(STEPS, tokens, n_in, generator=gen, device="cuda").to(torch.bfloat16)
    y = torch.zeros(STEPS, tokens, n_out, dtype=torch.bfloat16, device="cuda")
    rotated = torch.zeros(tokens, n_in, dtype=torch.bfloat16, device="cuda")
    splits = lin.tc_splits(n_out)
    z = torch.zeros(splits, tokens, n_out, device="cuda")
    torch.cuda.synchronize()
    for i in range(STEPS):
        lin.qtip_prepare(w, x[i], None, rotated, tokens)
        gpu.codec.swizzle_for_kernel(packed[i & 1], n_out, n_in, w.trellis)
        lin.qtip_multiply_batch(w, rotated, z, n_out, splits, tokens)
        lin.qtip_finish(w, z, y[i], None, False, splits, tokens)
    torch.cuda.synchronize()
    lin.kernel_status()
    return y


TOKENS = (1, 5, 9, 16, 64, 200)


def test_chained_launches_give_the_bits_of_plain_ones(gpu, tmp_path):
    out = str(tmp_path / "plain.pt")
    env = dict(os.environ, QTIP_PDL="0")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], env=env, cwd=ROOT, check=True, timeout=300)
    plain = torch.load(out)
    for tokens in TOKENS:
        for _ in range(3):
            assert torch.equal(decode_steps(gpu, tokens).cpu(), plain[tokens]), tokens


@pytest.mark.parametrize("tokens", [9, 96, 144])
def test_surplus_splits_under_capture(gpu, tokens):
    """More K-splits than cuts: the zero fill of the surplus slices and the chained product behind it, recorded and replayed."""
    lin, gen = gpu.linear, torch.Generator(device="cuda").manual_seed(tokens)
    n_in, n_out, splits = 128, 256, 4
    trellis = torch.randint(-32768, 32768, (n_in * n_out // 256 * 32,), generator=gen, device="cuda", dtype=torch.int16)
    one = torch.ones(n_out, device="cuda")
    w = lin.Matrix(trellis, one[:n_in], one, lin.runtime_lut(gpu.synth.seeded_tlut(1)), n_in, n_out)
    x = torch.randn(tokens, n_in, generator=gen, device="cuda").to(torch.bfloat16)
    want, z = torch.empty(splits, tokens, n_out, device="cuda"), torch.empty(splits, tokens, n_out, device="cuda")
    lin.qtip_multiply_tc(w, x, want, n_out, splits, tokens)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        lin.qtip_multiply_tc(w, x, z, n_out, splits, tokens)
        lin.qtip_multiply_tc(w, x, z, n_out, splits, tokens)
    for _ in range(3):
        z.fill_(float("nan"))
        graph.replay()
        assert torch.equal(z, want) and not bool(want[2:].any())


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    import __graft_entry__
    pkg = __graft_entry__.load_package()
    torch.save({t: decode_steps(pkg, t).cpu() for t in TOKENS}, sys.argv[1])
