"""The share of a dense K that stays in L2."""
import os
import subprocess

import pytest

from demystification_dfn_b200 import networks
from demystification_dfn_b200.ensemble import Ensemble
from demystification_dfn_b200.simulation import Simulation

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
MiB = 1 << 20
CHUNK = 4096

SRC = r"""
#include "kv_l2.cuh"
#include <cstdio>
#include <vector>
int main()
{
    // lines of: number of tiles, rows per tile
    std::vector<long long> rows;
    long long n, r;
    while (scanf("%lld %lld", &n, &r) == 2) rows.insert(rows.end(), (size_t)n, r);
    printf("%lld\n", (long long)l2_keep_tiles((int64_t)rows.size(), [&](int64_t i) { return (int64_t)rows[i] * 4096; }));
}
"""


@pytest.fixture(scope="module")
def keep(tmp_path_factory):
    d = tmp_path_factory.mktemp("l2")
    (d / "m.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "demystification_dfn_b200", "csrc"), "-o",
                    str(d / "m"), str(d / "m.cpp")], check=True)

    def run(*groups):
        text = "".join("%d %d\n" % g for g in groups)
        return int(subprocess.run([str(d / "m")], input=text, capture_output=True, text=True, check=True).stdout)

    return run


@pytest.mark.parametrize("groups,policy", [
    ([(0, 0)], False), ([(1, 8)], False), ([(160, 64)], False),
    ([(256, 64)], False),                      # 64 MiB: the largest that carries no policy
    ([(256, 64), (1, 1)], True),
    ([(500, 64)], True), ([(2861, 64)], True),
    ([(100, 128), (4000, 8)], True),           # tall tiles first, many short ones
    ([(4000, 8), (100, 128)], True),
    ([(20000, 1), (1, 128), (20000, 1)], True),
])
def test_kept_share_is_bounded_by_the_bytes_read(keep, groups, policy):
    """No policy for what fits in L2 as it is stored (padding included); of
    more than that the leading tiles up to 48 MiB, within one tile of it."""
    rows = [r for n, r in groups for _ in range(n)]
    k = keep(*groups)
    if not policy:
        assert sum(rows) * CHUNK <= 64 * MiB
        assert k == -1
        return
    assert 0 <= k < len(rows)
    kept = sum(rows[:k]) * CHUNK
    assert kept <= 48 * MiB < kept + rows[k] * CHUNK


@pytest.mark.gpu
def test_small_matrix_beside_a_kept_share():
    """K.V of 64 MiB, which L2 holds, before and after another handle has taken
    its kept share: 7.5 and 7.7 us, so at most 1.2 times (1.38 when the small
    matrix is copied at a lower priority than lines that carry none). The
    smallest of several runs on both sides."""
    def handle(n):
        return Simulation(networks.single_fault(n_el=n, length=10.0 * n, mode="modeII"), pressure="tridiag")

    with handle(2048) as small:
        alone = min(small.time_kernel(50) for _ in range(8))
        with handle(4000) as large:
            beside = 1e9
            for _ in range(8):
                large.time_kernel(20)
                beside = min(beside, small.time_kernel(50))
    assert beside <= 1.2 * alone


@pytest.mark.gpu
@pytest.mark.parametrize("mode,storage,n,count", [("modeII", "fp64", 4000, 1), ("modeIII", "bf16x2", 1500, 30)])
def test_kept_share_ends_with_the_handle(mode, storage, n, count):
    """Reads of a 90 MiB array, which L2 holds, before a handle with a kept
    share and after its end: alike, so at most 1.1 times (1.3 when the kept
    lines stay behind, which it takes about 75 reads to push out). The median
    of 25 reads on both sides, the best of three handles."""
    import torch

    x = torch.zeros(90 << 18, dtype=torch.float32, device="cuda")
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def reads():
        t = []
        for _ in range(25):
            a.record()
            x.sum()
            b.record()
            b.synchronize()
            t.append(a.elapsed_time(b))
        return sorted(t[2:])[11]

    other = torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    p = networks.single_fault(n_el=n, length=10.0 * n, mode=mode)
    ratios = []
    for _ in range(3):
        for k in range(4):
            other.fill_(k)      # whatever was kept before is gone
        reads()
        before = reads()
        e = Ensemble([p] * count, storage=storage, pressure="tridiag")
        e.time_kernel(20)
        e.close()
        ratios.append(reads() / before)
    assert min(ratios) <= 1.1, ratios
