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


def _largest_prime(below, step):
    """the largest prime = 1 (mod step) under `below`"""
    v = (below - 2) // step * step + 1
    while True:
        if all(pow(a, v - 1, v) == 1 for a in (2, 3, 5, 7, 11, 13)):
            return v
        v -= step


@pytest.mark.parametrize("log_n", [12, 14, 15, 17])
def test_prime_classes_at_their_upper_edges(log_n):
    """forward and inverse transforms with the largest primes of every arithmetic class (41, 50, 60 and 61 bits: the residues
    run up to the policies' bounds), on uniform input, all q - 1, all 0 and a single q - 1"""
    from oracle_lib import Oracle
    from pyPhantom._native import LIB, check
    N = 1 << log_n
    primes = [_largest_prime(1 << b, 2 * N) for b in (61, 50, 41, 60, 46)] + [_largest_prime((1 << 50) + (1 << 49), 2 * N)]
    parms = ph.params(ph.scheme_type.ckks)
    parms.set_poly_modulus_degree(N)
    parms.set_coeff_modulus(primes)
    parms.set_special_modulus_size(1)
    ctx, o = ph.context(parms), Oracle(N, primes, 1)
    q = np.array(primes, dtype=np.uint64)[:, None]
    spike = np.zeros((len(primes), N), dtype=np.uint64)
    spike[:, N - 1:] = q - np.uint64(1)
    for x in (o.fill(1, o.primes, 9, 50)[0], np.broadcast_to(q - np.uint64(1), spike.shape).copy(), spike):
        for call, want in ((LIB.b2_ntt_forward, o.ntt_forward(x)), (LIB.b2_ntt_inverse, o.ntt_inverse(x))):
            d = dev(x)
            check(call(ctx._h, d.data_ptr(), len(primes), 0, torch.cuda.current_stream().cuda_stream))
            assert np.array_equal(host(d), want)
