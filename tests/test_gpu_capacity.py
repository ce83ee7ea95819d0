"""A proteome with more seen (K-1)-mers than the scratch has count entries: the call reports
it, reads nothing outside its scratch, and the scratch serves the next call."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import oracle as O
from rocket_gb300 import _native
from rocket_gb300.kernels import CompositionVectorKernels

from gpu_helpers import to_device_bytes, ulp_diff

pytestmark = pytest.mark.gpu

AMINO = np.frombuffer(b"ACDEFGHIKLMNPQRSTVWY", np.uint8)


@pytest.mark.parametrize("k", [6, 7])
def test_more_seen_prefixes_than_count_entries(k):
    size, n = 1000, 5_000_000
    seq = AMINO[np.random.default_rng(k).integers(0, 20, n)].tobytes()
    # 2.5 M distinct 5-mers (4.9 M 6-mers) against 2 size + 2^20 entries of 8 bytes: at K = 6
    # the last of them would lie past the end of the scratch
    ker = CompositionVectorKernels("protein", k, size, n)
    keys = torch.full((size,), -1, dtype=torch.int32, device="cuda")
    vals = torch.zeros(size, dtype=torch.float32, device="cuda")
    with pytest.raises(_native.CudaException):
        ker.build_vector_gpu(to_device_bytes(seq), keys, vals, n)
    assert int((keys != -1).sum()) == 0  # nothing written
    short = seq[:60]
    m = ker.build_vector_gpu(to_device_bytes(short), keys, vals, len(short))
    want = O.cv_native(short, k, "protein")
    assert m == len(want["keys"])
    assert np.array_equal(keys.cpu().numpy().view(np.uint32)[:m], want["keys"])
    assert ulp_diff(vals.cpu().numpy()[:m], want["values"]) <= 1  # the builder's tests' bound
