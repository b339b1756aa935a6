"""Dispatch edges of the key switch over ring sizes, against the CPU oracle: which kernels a call runs depends on the ring,
the batch and the classes of the primes, the limbs do not."""
import numpy as np
import pytest
import torch

from gpu_helpers import dev, host, make_ctx

ph = pytest.importorskip("pyPhantom")
pytestmark = pytest.mark.gpu


def _key(ctx, digits):
    return ph.relin_key.from_numpy(ctx, digits)


@pytest.mark.parametrize("log_n,bits,special,l,batch", [
    (12, [60, 40, 40, 60], 1, 3, 2),                       # one limb per digit
    (14, [60, 40, 50, 36, 45, 60, 60], 2, 5, 3),           # every prime class, ragged last digit
    (15, [60, 40, 40, 40, 40, 60, 60], 2, 5, 2),           # 256-point rows behind a 128-point column pass
    (15, [60, 46, 40, 50, 60, 59, 60], 3, 2, 2),           # fewer limbs than a digit holds
    (17, [60, 40, 40, 60], 1, 2, 2),
])
def test_batched_products_equal_the_oracle(log_n, bits, special, l, batch):
    N = 1 << log_n
    ctx, o = make_ctx(N, bits, special)
    key = o.synth_key(o.beta(l), 4, 10)
    a, b = [o.synth_ct(l, 4, 20 + i) for i in range(batch)], [o.synth_ct(l, 4, 40 + i) for i in range(batch)]
    got = host(ph.multiply_relin_rescale_batch(ctx, dev(np.stack(a)), dev(np.stack(b)), _key(ctx, key)))
    for i in range(batch):
        assert np.array_equal(got[i], o.rescale(l, o.multiply_and_relin(l, a[i], b[i], key))), f"pair {i}"
    assert ctx.device_status() == 0
