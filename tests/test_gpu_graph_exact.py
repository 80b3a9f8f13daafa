"""GPU: a graph batch (BC_BATCH_GRAPH) that follows one of the same lengths but
another number of products (a cluster each, a block each) gives exact products;
its outputs are cleared before every call."""
import numpy as np
import pytest

from conftest import exact, limbs

pytestmark = pytest.mark.gpu


def test_exact_products_as_the_kernels_change(gpu):
    torch = pytest.importorskip("torch")
    for k, n in enumerate((20, 400, 20, 400)):
        al, bl = 230, 215
        pool = limbs(31 * k + 1, n * (al + bl))
        dev = torch.from_numpy(pool.view(np.int32)).cuda()
        out = torch.zeros(n * (al + bl), dtype=torch.int32, device="cuda")
        descs = (gpu.MulDesc * n)()
        for i in range(n):
            o = 4 * i * (al + bl)
            descs[i] = gpu.MulDesc(out.data_ptr() + o, al + bl, dev.data_ptr() + o, al, dev.data_ptr() + o + 4 * al, bl)
        st = gpu.mul_batch_desc(descs, n, gpu.BATCH_GRAPH)
        assert st["graph_launches"] == 1
        got = out.cpu().numpy().view(np.uint32).reshape(n, al + bl)
        for x, c in zip(pool.reshape(n, al + bl), got):
            assert np.array_equal(c, exact(x[:al], x[al:], al + bl)), (k, n)
