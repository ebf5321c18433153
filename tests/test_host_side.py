"""CPU checks of the package's host half."""
import subprocess
import sys

import pytest
import torch

from conftest import REPO


def test_native_module_is_loaded_with_the_cache():
    """Not inside a process's first decode step."""
    code = ("from shard_b200 import _lib, Cache, build; build.build(); Cache(num_layers=1); assert _lib._host is not None")
    subprocess.run([sys.executable, "-c", code], cwd=REPO, check=True)


def test_a_cache_can_be_made_without_the_native_module(monkeypatch):
    from shard_b200 import Cache, _lib

    def missing():
        raise _lib.ShardError("not built")

    monkeypatch.setattr(_lib, "host", missing)
    assert Cache(num_layers=2).get_seq_length() == 0


def _allocation(variances, budget):
    """The dynamic programme of the reference, table by table."""
    v = variances.float()
    sizes = [min(64, len(v) - i) for i in range(0, len(v), 64)]
    var = [v[64 * g:64 * g + s].sum().item() for g, s in enumerate(sizes)]
    cap = budget // 16 + 1
    best = [[0.0] * (cap + 1)] + [[float("inf")] * (cap + 1) for _ in sizes]
    pick = [[0] * (cap + 1) for _ in range(len(sizes) + 1)]
    cost = [{b: (s * b + 15) // 16 for b in (0, 2, 4, 6, 8)} for s in sizes]
    for g in range(len(sizes)):
        for b in range(cap + 1):
            for bits, c in cost[g].items():
                if c <= b:
                    total = best[g][b - c] + (var[g] * 4 if bits == 0 else var[g] / (3.0 * 4 ** bits))
                    if total < best[g + 1][b]:
                        best[g + 1][b], pick[g + 1][b] = total, bits
    b = min(range(cap + 1), key=lambda i: best[-1][i])
    out = [0] * len(sizes)
    for g in reversed(range(len(sizes))):
        out[g] = pick[g + 1][b]
        b -= cost[g][out[g]]
    return [bits for bits, s in zip(out, sizes) for _ in range(s)]


@pytest.mark.parametrize("d,budget", [(192, 819), (1, 64), (64, 0), (65, -1), (200, -16), (5000, 3000), (4097, 40000), (100, 5000)])
def test_bit_allocation(d, budget):
    """Any number of components and any budget the programme can be asked for."""
    from shard_b200.rope import dp_bit_allocation
    v = torch.exp(-0.01 * torch.arange(d)) * (1 + 0.3 * torch.rand(d, generator=torch.Generator().manual_seed(d)))
    assert dp_bit_allocation(v, budget) == _allocation(v, budget)
    for odd in (float("nan"), float("inf")):
        w = v.clone()
        w[d // 2] = odd
        assert dp_bit_allocation(w, budget) == _allocation(w, budget)


def test_bit_allocation_ends():
    from shard_b200._lib import ShardError
    from shard_b200.rope import dp_bit_allocation
    assert dp_bit_allocation(torch.zeros(0), 100) == []
    v = torch.rand(300, generator=torch.Generator().manual_seed(1))
    assert dp_bit_allocation(v, 1 << 40) == dp_bit_allocation(v, 1 << 20) == _allocation(v, 10000) == [8] * 300
    with pytest.raises(ShardError):
        dp_bit_allocation(v, -17)
    with pytest.raises(TypeError):
        dp_bit_allocation(v, 100.5)


def test_stream_signs_are_the_callers():
    """Every call gives a tensor of its own."""
    from shard_b200.streaming import stream_signs
    a, b = stream_signs(3, 128, "cpu"), stream_signs(3, 128, "cpu")
    a.zero_()
    assert bool((b.abs() == 1).all()) and torch.equal(b, stream_signs(3, 128, "cpu"))


@pytest.mark.parametrize("before,during", [(3, 0), (3, 2), (0, 4)])
def test_the_clock_record_says_what_it_was_sampled_in(tmp_path, before, during):
    """Samples of the timed region count; where there are none the last one from before it stands in, and the record says so."""
    import bench
    sampler = bench.ClockSampler(0)
    sampler.path = str(tmp_path / "clocks.csv")
    sampler.proc = subprocess.Popen([sys.executable, "-c", ""])
    idle, busy = "120, 1965, 200.0, Not Active, Not Active, Not Active, Not Active\n", "1965, 1965, 700.0, Not Active, Not Active, Not Active, Active\n"
    with open(sampler.path, "w") as f:
        f.write(idle * before)
    sampler.mark()
    with open(sampler.path, "a") as f:
        f.write(busy * during)
    got = sampler.stop()
    assert got["samples"] == during and got["sm_mhz"] == (1965 if during else 120)
    assert ("note" in got) == (during == 0)
    assert got["reasons"] == (["sw_power_cap"] if during else [])
