"""GPU parity of successive graph batches (BC_BATCH_GRAPH) of one launch
structure but other kernels: products of one length run a cluster each while
they are few and a block each when they are many, and a length's outer pass
reads one or two pieces of the operands.  Every output must equal the plain
batch's, and the kept executable graph must be renewed when a kernel changes
and kept when none does."""
import numpy as np
import pytest

from conftest import limbs

pytestmark = pytest.mark.gpu


def _batch(gpu, torch, n, al, bl, seed):
    pool = torch.from_numpy(limbs(seed, n * (al + bl)).view(np.int32)).cuda()
    out = torch.zeros(n * (al + bl), dtype=torch.int32, device="cuda")
    descs = (gpu.MulDesc * n)()
    for i in range(n):
        a = pool.data_ptr() + 4 * i * (al + bl)
        descs[i] = gpu.MulDesc(out.data_ptr() + 4 * i * (al + bl), al + bl, a, al, a + 4 * al, bl)
    return descs, pool, out


@pytest.mark.parametrize("steps", [
    # (products, AL, BL): a cluster each, a block each, a cluster each again
    [(20, 230, 230), (400, 230, 230), (20, 230, 230)],
    [(400, 230, 230), (20, 230, 230), (20, 231, 229)],
    # long and short operands of one sum, then small products
    [(3, 40_000, 40_000), (3, 70_000, 10_000), (2, 300, 300), (300, 300, 300)],
])
def test_graph_renewed_when_a_kernel_changes(gpu, steps):
    torch = pytest.importorskip("torch")
    for k, (n, al, bl) in enumerate(steps):
        descs, pool, out = _batch(gpu, torch, n, al, bl, 12_000 + 10 * k)
        gpu.mul_batch_desc(descs, n)
        torch.cuda.synchronize()
        plain = out.clone()
        for again in range(2):
            out.zero_()
            st = gpu.mul_batch_desc(descs, n, gpu.BATCH_GRAPH)
            torch.cuda.synchronize()
            assert st["graph_launches"] == 1
            assert torch.equal(out, plain)
            if again:
                assert st["graph_updates"] == 1  # the same kernels: updated in place
            elif k and n != steps[k - 1][0]:
                assert st["graph_updates"] == 0  # clusters or not: a new graph
