"""GPU test of the one-launch copy of many arrays: sizes around its 16-byte words and 16 KB
tiles, ends on any byte, more arrays than one launch takes, and pairs it leaves to torch."""
import numpy as np
import pytest

from clmgb.state import copy_arrays

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 127, 128, 129, 300])
def test_copies_every_byte_and_no_other(count):
    rng = np.random.default_rng(count)
    sizes = [0, 1, 15, 16, 17, 255, 16383, 16384, 16385, 40000]
    pairs, want = [], []
    for i in range(count):
        n, od, os_ = int(rng.choice(sizes)), int(rng.choice([0, 1, 8, 16])), int(rng.choice([0, 1, 8, 16]))
        src = torch.from_numpy(rng.integers(0, 256, n + 40, dtype=np.uint8)).cuda()
        dst = torch.full((n + 40,), 7, dtype=torch.uint8, device="cuda")
        w = dst.clone()
        w[od:od + n] = src[os_:os_ + n]
        pairs.append((dst[od:od + n], src[os_:os_ + n]))
        want.append((dst, w))
    copy_arrays(pairs)
    for d, w in want:
        assert torch.equal(d, w)


def test_other_pairs():
    a = torch.randn(50, 30, device="cuda", dtype=torch.float64)
    b, c, d = torch.empty(30, 50, device="cuda", dtype=torch.float64), torch.empty(50, 30, device="cuda"), torch.empty(50, 30)
    copy_arrays([(b, a.t()), (c, a), (d, a), (a, a)])
    assert torch.equal(b, a.t()) and torch.equal(c, a.float()) and torch.equal(d, a.float().cpu())
