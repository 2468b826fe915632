"""A tuning cache written for other kernels is not used."""
import pytest

import afmm2d_b200 as A
from afmm2d_b200 import workloads


@pytest.mark.gpu
def test_entries_of_earlier_kernels_miss(tmp_path):
    pts, _, _ = workloads.make("mixture4m", N=16384)
    a = A.AFMM(16384, 64, 6, pts, kernel="one_over_r")
    a.assemble()
    cache = tmp_path / "tuning.txt"
    assert not a.autotune(cache=cache)[1]
    key = cache.read_text().split()[0]
    fields = key.split("|")
    n = len("kernels=")
    earlier = ["|".join(f for f in fields if not f.startswith("kernels=")),  # as written before there was a version
               "|".join(f[:n] + "1" if f.startswith("kernels=") else f for f in fields)]
    for k in earlier:
        assert k != key
        old = tmp_path / "old.txt"
        old.write_text(f"{k} 32768 0 3 3 16 1 0 0\n")
        b = A.AFMM(16384, 64, 6, pts, kernel="one_over_r")
        b.assemble()
        hit = b.autotune(cache=old)[1]
        assert not hit and len(old.read_text().splitlines()) == 2
        assert b.autotune(cache=old)[1]  # its own entry is found
