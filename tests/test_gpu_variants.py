"""GPU: the kernels behind a choice on sizes or structure, each at the sizes
where that choice can go wrong, against the CPU oracle (or plain numpy / FP64
torch where the oracle has no such function)."""
import numpy as np
import pytest

from isai_kernel_gb300 import gen

pytestmark = pytest.mark.gpu


def T(a, dev):
    import torch

    return torch.from_numpy(np.ascontiguousarray(a)).to(dev)


def N(t):
    return t.detach().cpu().numpy()


def scalar_csr(rng, nb, bs, most, shuffled):
    """A scalar CSR matrix of nb*bs rows with up to `most` entries a row, some
    rows empty, some columns repeated; `shuffled` leaves every third row's
    entries in random order."""
    n = nb * bs
    rows = []
    for i in range(n):
        k = 0 if rng.random() < 0.15 else int(rng.integers(0, most + 1))
        c = rng.integers(0, n, size=k)
        if k > 2 and rng.random() < 0.5:
            c[1] = c[0]
        c = c if shuffled and i % 3 == 0 else np.sort(c)
        rows.append(c.astype(np.int32))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum([len(c) for c in rows], out=rp[1:])
    col = np.concatenate(rows) if n else np.zeros(0, np.int32)
    return rp, col, rng.uniform(-1, 1, size=col.shape[0])


# Bit for bit: the block columns are integers and every scalar position sums
# its entries in file order in both.
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("nb", [1, 3, 33])
@pytest.mark.parametrize("bs", [1, 2, 3, 4, 5, 6, 7, 8])
def test_csr_to_bsr_merge(cuda, orc, bs, nb, shuffled):
    from isai_kernel_gb300 import api

    rng = np.random.default_rng(100 * bs + nb)
    rp, col, val = scalar_csr(rng, nb, bs, 12 if nb < 33 else 70, shuffled)
    _, r, c, v = api.csr_to_bsr5(nb * bs, bs, T(rp, cuda), T(col, cuda), T(val, cuda))
    ro, co, vo = orc.csr_to_bsr(nb * bs, bs, rp, col, val)
    assert np.array_equal(N(r), ro) and np.array_equal(N(c), co)
    assert np.array_equal(N(v), vo)


@pytest.mark.parametrize("bad", [-1, 40])
def test_csr_to_bsr_column_out_of_range(cuda, bad):
    from isai_kernel_gb300 import api

    rp = np.arange(0, 81, 2, dtype=np.int32)
    col = np.tile(np.array([0, 39], np.int32), 40)
    col[50] = bad
    with pytest.raises(api.BiluError):
        api.csr_to_bsr5(40, 5, T(rp, cuda), T(col, cuda), T(np.ones(80), cuda))
