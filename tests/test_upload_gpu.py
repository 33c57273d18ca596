"""Uploads of pageable arrays through the staging threads: every byte arrives,
from several threads and streams at once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# below and above the staging size (16 MB), chunk edges (1 MB) with remainders;
# pinned sources take the plain copy
@pytest.mark.parametrize("nbytes", [1, 16 * 2**20 - 1, 16 * 2**20, 16 * 2**20 + 1,
                                    17 * 2**20 + 12345, 64 * 2**20])
@pytest.mark.parametrize("pinned", [False, True])
def test_upload(nbytes, pinned):
    import torch

    from mlxlearn_b200 import _lib
    from mlxlearn_b200.index import build_index

    index = build_index(np.eye(8, dtype=np.float32))
    index._ensure_device()
    failures = []

    def one(i):
        src = torch.empty(nbytes, dtype=torch.uint8, pin_memory=pinned).numpy()
        part = np.random.default_rng(nbytes + i).integers(0, 256, 1 + nbytes // 97, dtype=np.uint8)
        src[:] = part.repeat(97)[:nbytes]
        src[-1] = i
        want = src.copy()
        stream = torch.cuda.Stream()
        dst = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        rc = _lib.load().b2k_upload(dst.data_ptr(), src.ctypes.data, nbytes, stream.cuda_stream)
        if not pinned:
            src[:] = 0  # the source is free on return
        stream.synchronize()
        if rc or not np.array_equal(dst.cpu().numpy(), want):
            failures.append(i)

    one(0)
    threads = [threading.Thread(target=one, args=(i,)) for i in range(1, 4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
    index.close()
