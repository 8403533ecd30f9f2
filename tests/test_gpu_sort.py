"""The Morton-code sort at the edges of its forms: one cluster of blocks up to 16,384 keys (1 or 4 keys per
thread), one-sweep passes of 4,096-key tiles above. Keys and the stable permutation must equal numpy's stable argsort."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def keys_of(kind, n, rng):
    if kind == "random":
        return rng.integers(0, 1 << 64, n, dtype=np.uint64, endpoint=False)
    if kind == "few":  # three distinct keys, constant digits between them
        return rng.choice(np.array([5, 5 << 40, (1 << 64) - 1], np.uint64), n)
    if kind == "equal":
        return np.full(n, 0x0123456789ABCDEF, np.uint64)
    return np.sort(rng.integers(0, 1 << 63, n, dtype=np.uint64))[::-1].copy()  # descending


@pytest.mark.parametrize("n", [1, 2, 33, 1023, 1024, 1025, 4096, 4097, 8191, 8193, 16383, 16384, 16385, 20479, 20480, 20481, 300001])
@pytest.mark.parametrize("kind", ["random", "few", "equal", "descending"])
@pytest.mark.parametrize("in_place", [False, True])
def test_sort_codes(nb, n, kind, in_place):
    import torch

    k = keys_of(kind, n, np.random.default_rng(n))
    order = np.argsort(k, kind="stable")
    src = torch.from_numpy(k.view(np.int64)).cuda()
    dst = src if in_place else torch.empty_like(src)
    ids = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    rc = nb.lib().nb_sort_codes_noalloc(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()),
                                        C.c_void_p(ids.data_ptr()), n, None)
    assert rc == nb.NB_OK
    assert np.array_equal(dst.cpu().numpy().view(np.uint64), k[order])
    assert np.array_equal(ids.cpu().numpy().astype(np.int64), order)
