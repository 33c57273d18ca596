"""What b2k_upload promises: the source may be reused on return whatever memory it
is, and the copy is ordered on the caller's stream, the per-thread one included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread


@pytest.fixture
def index():
    from mlxlearn_b200.index import build_index

    index = build_index(np.eye(8, dtype=np.float32))
    index._ensure_device()  # staging threads run while an index lives
    yield index
    index.close()


# below and above the size from which pageable memory is staged (16 MB)
@pytest.mark.parametrize("nbytes", [1000, 3 * 2**20, 33 * 2**20 + 5])
@pytest.mark.parametrize("memory", ["pageable", "pinned"])
@pytest.mark.parametrize("stream", ["own", "per_thread", "legacy"])
def test_source_is_free_and_stream_order_holds(index, nbytes, memory, stream):
    import torch

    from mlxlearn_b200 import _lib

    src = torch.empty(nbytes, dtype=torch.uint8, pin_memory=memory == "pinned").numpy()
    src[:] = np.random.default_rng(nbytes).integers(1, 256, nbytes, dtype=np.uint8)
    want = src.copy()
    dst = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    s = {"own": torch.cuda.Stream(), "per_thread": torch.cuda.ExternalStream(PER_THREAD),
         "legacy": torch.cuda.default_stream()}[stream]
    with torch.cuda.stream(s):
        torch.cuda._sleep(40_000_000)  # about 20 ms: the copy waits behind it
        dst.zero_()
    rc = _lib.load().b2k_upload(dst.data_ptr(), src.ctypes.data, nbytes, s.cuda_stream)
    src[:] = 0
    s.synchronize()
    assert rc == 0
    assert np.array_equal(dst.cpu().numpy(), want)
