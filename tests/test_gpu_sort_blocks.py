"""Sorts on both sides of the block sizes of a pass (4, 8 and 15 rows), by an even and an odd number of
passes, with live counts at block edges, sizes in turn on one scratch whose flag arena grows and shrinks:
stable order of keys and values."""
import pytest

pytestmark = pytest.mark.gpu

SIZES = [65_537, 67_584, 67_585, 196_608, 196_609, 200_705, 1_638_400, 1_638_401]


def _check(gs, torch, n, live, key_bits, scratch, nbytes, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    keys = torch.randint(0, 1 << 31, (n,), generator=g, device="cuda")
    keys = (keys * 2 + torch.randint(0, 2, (n,), generator=g, device="cuda")) & ((1 << key_bits) - 1)
    keys[::5] = keys[0]  # runs of equal keys
    values = torch.arange(n, device="cuda", dtype=torch.int32)
    k = (((keys + (1 << 31)) & 0xFFFFFFFF) - (1 << 31)).int()  # the same 32 bits
    v, count = values.clone(), torch.tensor([live], dtype=torch.int32, device="cuda")
    before = k.clone()
    gs.RadixSorter.sort(k, v, n, scratch, nbytes, count=count, key_bits=key_bits)
    torch.cuda.synchronize()
    order = torch.sort(keys[:live], stable=True).indices
    assert torch.equal(k[:live], before[:live][order]) and torch.equal(v[:live], values[:live][order])
    assert torch.equal(k[live:], before[live:]) and torch.equal(v[live:], values[live:])


@pytest.mark.parametrize("key_bits", [32, 30, 24, 16])
@pytest.mark.parametrize("n", SIZES)
def test_block_sizes(gs, cuda, n, key_bits):
    nbytes = gs.RadixSorter.scratch_bytes(n)
    scratch = cuda.zeros(nbytes, dtype=cuda.uint8, device="cuda")
    for live in (n, n // 2, 2048, 1, 0):
        _check(gs, cuda, n, live, key_bits, scratch, nbytes, seed=n + live)


def test_block_sizes_in_turn(gs, cuda):
    nbytes = gs.RadixSorter.scratch_bytes(1_700_000)
    scratch = cuda.zeros(nbytes, dtype=cuda.uint8, device="cuda")
    for i, n in enumerate([100_000, 1_700_000, 150_000, 400_000, 30_000, 1_600_000, 100_000, 1_650_000]):
        for key_bits in (30, 32):
            _check(gs, cuda, n, n - 7 * i, key_bits, scratch, nbytes, seed=i)


@pytest.mark.parametrize("key_bits", [9, 12, 13, 16, 30, 32])
@pytest.mark.parametrize("n", [65_537, 196_608, 1_000_001])
def test_smallest_accepted_scratch(gs, cuda, n, key_bits):
    """With the fewest bytes of scratch that the entry point accepts, nothing beyond them is written."""
    full = gs.RadixSorter.scratch_bytes(n)
    keys = cuda.zeros(n, dtype=cuda.int32, device="cuda")
    count = cuda.zeros(1, dtype=cuda.int32, device="cuda")
    scratch = cuda.zeros(full + 65_536, dtype=cuda.uint8, device="cuda")

    def accepted(nbytes):
        try:
            gs.RadixSorter.sort(keys, keys.clone(), n, scratch, nbytes, count=count, key_bits=key_bits)
        except gs.GsError:
            return False
        return True

    lo, hi = 0, full  # refused, accepted
    while hi - lo > 1:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if accepted(mid) else (mid, hi)
    cuda.cuda.synchronize()
    scratch[hi:] = 0xA5
    scratch[:hi] = 0
    for live in (n, n // 3):
        _check(gs, cuda, n, live, key_bits, scratch, hi, seed=n + key_bits)
    assert bool((scratch[hi:] == 0xA5).all())
