"""The trace calls' device scratch (GPU): the tap tables of a batch of many
distinct lengths go back to the driver with the call, and the envelopes of the
next, ordinary call are the same before and after."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_large_tap_tables_are_given_back():
    import torch
    from pefdtd import traces
    rng = np.random.default_rng(0)
    small = [rng.normal(size=n) for n in (400, 401, 900)]
    first = traces.envelope(small)
    many = [rng.normal(size=20000 + k) for k in range(300)]   # 48 MB of taps
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free0 = torch.cuda.mem_get_info()[0]
    env = traces.envelope(many)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    assert free0 - torch.cuda.mem_get_info()[0] <= 16 << 20
    for x, e in zip(many[::100], env[::100]):
        n = len(x)
        h = np.zeros(n)
        h[0] = 1
        h[1:(n + 1) // 2] = 2
        if n % 2 == 0:
            h[n // 2] = 1
        ref = np.abs(np.fft.ifft(np.fft.fft(x) * h))
        # n products of size 1 / k each: rounding grows no faster than n eps
        assert np.abs(e - ref).max() <= n * 2.3e-16 * np.abs(ref).max()
    for a, b in zip(first, traces.envelope(small)):
        assert np.array_equal(a, b)
