"""The sorter at the sizes where it changes between one cluster (1, 2 or 4 rows a thread, 1 to 16
CTAs) and the pass kernels, with device-side counts below the capacity, keys of all ones (the padding's
value) and ties, against a stable sort: equal bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 33, 1023, 1024, 1025, 16_384, 16_385, 32_768, 32_769, 65_536, 65_537, 131_072, 131_073]


@pytest.mark.parametrize("key_bits", [1, 8, 9, 30, 32])
@pytest.mark.parametrize("n", SIZES)
def test_cluster_sizes_counts_and_ties(gs, cuda, n, key_bits):
    torch = cuda
    rng = np.random.default_rng(n + key_bits)
    nbytes = gs.RadixSorter.scratch_bytes(n)
    scratch = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    for live in {n, n - 1, n // 2, 1, 0}:
        keys = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
        keys[rng.integers(0, n, size=n // 4)] = 0xFFFFFFFF
        keys[rng.integers(0, n, size=n // 4)] = keys[0]
        vals = rng.permutation(n).astype(np.uint32)
        pad = 64
        dk = torch.full((n + pad,), -7, dtype=torch.int32, device="cuda")
        dv = torch.full((n + pad,), -7, dtype=torch.int32, device="cuda")
        dk[:n] = torch.from_numpy(keys.view(np.int32)).cuda()
        dv[:n] = torch.from_numpy(vals.view(np.int32)).cuda()
        count = torch.tensor([live], dtype=torch.int32, device="cuda")
        gs.RadixSorter.sort(dk, dv, n, scratch, nbytes, count=count, key_bits=key_bits)
        st, _ = gs.Renderer.status(scratch)
        assert st == 0
        m = np.uint64((1 << key_bits) - 1)
        order = np.argsort(keys[:live].astype(np.uint64) & m, kind="stable")
        got_k, got_v = dk.cpu().numpy().view(np.uint32), dv.cpu().numpy().view(np.uint32)
        assert np.array_equal(got_k[:live], keys[:live][order]) and np.array_equal(got_v[:live], vals[:live][order])
        assert np.array_equal(got_k[live:n], keys[live:]) and np.array_equal(got_v[live:n], vals[live:])
        assert (dk[n:] == -7).all() and (dv[n:] == -7).all()
