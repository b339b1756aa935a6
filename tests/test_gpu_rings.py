"""Dispatch edges of the key switch over ring sizes, against the CPU oracle: which kernels a call runs depends on the ring,
the batch and the classes of the primes, the limbs do not."""
import numpy as np
import pytest
import torch

from gpu_helpers import dev, host, kernels_of, make_ctx

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


@pytest.mark.parametrize("log_n,bits,special,l,n_steps", [
    (12, [60, 40, 50, 45, 60], 1, 3, 19),                  # more steps than one launch takes, one limb per digit
    (13, [60, 40, 36, 50, 40, 60, 59], 2, 5, 3),           # ragged last digit, every prime class
    (16, [60, 40, 40, 60, 60], 2, 3, 5),                   # chunks bounded by the L2
])
def test_hoisted_rotations_equal_the_oracle(log_n, bits, special, l, n_steps):
    """one result per step, their sum, and a result on top of its operand"""
    N = 1 << log_n
    steps = list(range(1, n_steps + 1))
    elts = [ph.get_elt_from_step(s, N) for s in steps]
    ctx, o = make_ctx(N, bits, special, elts)
    keys = [o.synth_key(o.beta(l), 6, 100 + 40 * i) for i in range(n_steps)]
    glk = ph.galois_key.from_keys([ph.relin_key.from_numpy(ctx, k) for k in keys])
    ct_h = o.synth_ct(l, 6, 1)
    chain = o.size_Q - l + 1
    ct = ph.ciphertext.from_numpy(ctx, ct_h, chain)
    for got, want in zip(ph.hoist_rotations(ctx, ct, glk, steps), o.hoist_rotations(l, ct_h, elts, keys)):
        assert np.array_equal(got.numpy(), want)
    assert np.array_equal(ph.hoisting(ctx, ct, glk, steps).numpy(), o.hoisting_sum(l, ct_h, elts, keys))
    from pyPhantom import _native
    from pyPhantom._native import LIB, check
    s, tab = torch.cuda.current_stream().cuda_stream, glk.relin_keys[0].pointer_table()
    want = o.apply_galois(l, elts[0], keys[0], ct_h)
    for out in (ctx.empty(2, l), dev(ct_h)):
        src = out if out.data_ptr() != ct.data.data_ptr() and np.array_equal(host(out), ct_h) else ct.data
        ws, nb = ctx.workspace(_native.OP_ROTATE, l)
        check(LIB.b2_apply_galois(ctx._h, l, elts[0], src.data_ptr(), tab.ctypes.data, len(tab), out.data_ptr(), ws.data_ptr(), nb, s))
        assert np.array_equal(host(out), want)
    out = dev(ct_h)
    ws, nb = ctx.workspace(_native.OP_HOIST, l)
    ptr = np.array([out.data_ptr()], dtype=np.uint64)
    e0 = np.array(elts[:1], dtype=np.uint32)
    check(LIB.b2_hoist_rotations(ctx._h, l, out.data_ptr(), e0.ctypes.data, 1, tab.ctypes.data, len(tab), ptr.ctypes.data, ws.data_ptr(), nb, s))
    assert np.array_equal(host(out), o.hoist_rotations(l, ct_h, elts[:1], keys[:1])[0])
    assert ctx.device_status() == 0


@pytest.mark.parametrize("M", [1, 3, 64, 131])
def test_giant_steps_on_every_prime_class(M):
    """the sums of M products at the edges of their loops (groups of four, tables of 64, sums that have to be folded), operands
    at q - 1 so that every term is as large as it gets"""
    from oracle_lib import Oracle
    from pyPhantom._native import LIB, check
    N = 4096
    primes = [_largest_prime(1 << b, 2 * N) for b in (61, 60, 50, 41, 30)] + [_largest_prime((1 << 58) + 1, 2 * N)]
    parms = ph.params(ph.scheme_type.ckks)
    parms.set_poly_modulus_degree(N)
    parms.set_coeff_modulus(primes)
    parms.set_special_modulus_size(1)
    ctx, o, l = ph.context(parms), Oracle(N, primes, 1), 5
    q = np.array(primes[:l], dtype=np.uint64)[:, None]
    pts = [o.fill(1, o.primes[:l], 2, 10 + i)[0] for i in range(M)]
    bab = [o.synth_ct(l, 2, 500 + i) for i in range(M)]
    for i in range(M):
        pts[i][:, : N // 2] = q - np.uint64(1)
        bab[i][:, :, : N // 2] = q - np.uint64(1)
    want = o.bsgs_mac(l, pts, bab)
    dp, db = [dev(p) for p in pts], [dev(b) for b in bab]
    table = lambda ts: torch.tensor([t.data_ptr() for t in ts], dtype=torch.int64, device="cuda")
    s, tp, tb = torch.cuda.current_stream().cuda_stream, table(dp), table(db)
    out = ctx.empty(2, l)
    check(LIB.b2_bsgs_mac(ctx._h, l, M, tp.data_ptr(), tb.data_ptr(), out.data_ptr(), s))
    assert np.array_equal(host(out), want)
    for n in (2, 3, 4):
        outs = [ctx.empty(2, l) for _ in range(n)]
        tabs = torch.cat([tp] * n), table(outs)
        check(LIB.b2_bsgs_mac_multi(ctx._h, l, M, n, tabs[0].data_ptr(), tb.data_ptr(), tabs[1].data_ptr(), s))
        for t in outs:
            assert np.array_equal(host(t), want)


@pytest.mark.parametrize("log_n,l,batch", [(12, 3, 3), (15, 4, 2), (16, 3, 2)])
def test_batched_rotation_and_rotation_on_top_of_a_sum(log_n, l, batch):
    """b2_apply_galois_batch with gaps between the sets, and b2_rotate_add, against the oracle's rotations"""
    from pyPhantom import _native
    from pyPhantom._native import LIB, check
    N = 1 << log_n
    elt = ph.get_elt_from_step(3, N)
    ctx, o = make_ctx(N, [60, 40, 50, 40, 60, 60], 2, [elt])
    key = o.synth_key(o.beta(l), 8, 10)
    rk = ph.relin_key.from_numpy(ctx, key)
    tab, s = rk.pointer_table(), torch.cuda.current_stream().cuda_stream
    cts = [o.synth_ct(l, 8, 20 + i) for i in range(batch)]
    src = torch.zeros(batch, 2 * l + 1, N, dtype=torch.int64, device="cuda")
    for i, c in enumerate(cts):
        src[i, : 2 * l] = dev(c).reshape(2 * l, N)
    out = torch.zeros(batch, 2 * l + 2, N, dtype=torch.int64, device="cuda")
    ws = ph.keyswitch_batch_workspace(ctx, l, batch)
    check(LIB.b2_apply_galois_batch(ctx._h, l, elt, batch, src.data_ptr(), 2 * l + 1, tab.ctypes.data, len(tab), out.data_ptr(), 2 * l + 2,
                                    ws.data_ptr(), ws.numel() * 8, s))
    want = [o.apply_galois(l, elt, key, c) for c in cts]
    for i in range(batch):
        assert np.array_equal(host(out[i, : 2 * l]).reshape(2, l, N), want[i])
    assert not out[:, 2 * l:].any()
    acc = dev(cts[1])
    w1, nb = ctx.workspace(_native.OP_KEYSWITCH, l)
    check(LIB.b2_rotate_add(ctx._h, l, elt, dev(cts[0]).data_ptr(), tab.ctypes.data, len(tab), acc.data_ptr(), w1.data_ptr(), nb, s))
    assert np.array_equal(host(acc), np.stack([o.add(cts[1][k], want[0][k]) for k in range(2)]))


def test_product_with_diagonals_outside_pinned_memory():
    """the matrix product reads pinned diagonals in place; pageable ones are copied first and give the same limbs"""
    N, l, M, G = 4096, 3, 4, 5
    ctx, o = make_ctx(N, [60, 40, 40, 60], 1, [ph.get_elt_from_step(s, N) for s in (1, 2, 4)])
    glk = ph.galois_key.from_keys([ph.relin_key.from_numpy(ctx, o.synth_key(o.beta(l), 3, 10 + 20 * i)) for i in range(3)])
    coeffs = [o.synth_signed(5, 70 + d) for d in range(M * G)]
    x = ph.ciphertext.from_numpy(ctx, o.synth_ct(l, 3, 1), 1, 2.0 ** 40)
    pinned = ph.bsgs_diagonals([ph.single_chain_plaintext(c, 2.0 ** 40) for c in coeffs], M * G, M, G)
    plain = ph.bsgs_diagonals([ph.single_chain_plaintext(c, 2.0 ** 40) for c in coeffs], M * G, M, G)
    for p in plain.diagonals:
        p.coeffs = p.coeffs.clone()
    assert not plain.diagonals[0].coeffs.is_pinned()
    assert torch.equal(ph.bsgs_matmul_preencoded(ctx, glk, x, pinned).data, ph.bsgs_matmul_preencoded(ctx, glk, x, plain).data)


@pytest.mark.parametrize("log_n,bits,special,l,n", [
    (12, [60, 40, 50, 45, 60], 1, 3, 19),                  # more ciphertexts than one launch takes, the elements repeat
    (14, [60, 40, 36, 50, 40, 60, 59], 2, 5, 3),
    (15, [60, 40, 40, 60, 60], 2, 3, 1),
])
def test_sum_of_rotated_ciphertexts(log_n, bits, special, l, n):
    """b2_rotate_sum, alone and on top of a sum, against the oracle's stages: inner products added, one ModDown"""
    from pyPhantom._native import LIB, check
    N, n_elt = 1 << log_n, 3
    elts = [ph.get_elt_from_step(s, N) for s in range(1, n_elt + 1)]
    ctx, o = make_ctx(N, bits, special, elts)
    keys = [o.synth_key(o.beta(l), 8, 10 + 40 * i) for i in range(n_elt)]
    rks = [ph.relin_key.from_numpy(ctx, k) for k in keys]
    cts = [o.synth_ct(l, 8, 200 + i) for i in range(n)]
    q = np.concatenate([o.primes[:l], o.primes[-special:]])[None, :, None]
    add = lambda x, y, m: (x + y) % m                      # residues are below 2^61
    cx, c0 = 0, 0
    for i, ct in enumerate(cts):
        turned = ct[:, :, o.galois_perm(elts[i % n_elt])]
        cx = add(o.ks_inner_prod(l, o.modup(l, turned[1]), keys[i % n_elt]), cx, q)
        c0 = add(turned[0], c0, q[0, :l])
    want = np.stack([o.moddown(l, cx[k]) for k in range(2)])
    want[0] = add(want[0], c0, q[0, :l])
    src = torch.zeros(n, 2 * l + 1, N, dtype=torch.int64, device="cuda")
    for i, c in enumerate(cts):
        src[i, : 2 * l] = dev(c).reshape(2 * l, N)
    tab = np.concatenate([rks[i % n_elt].pointer_table() for i in range(n)])
    e = np.array([elts[i % n_elt] for i in range(n)], dtype=np.uint32)
    nb = int(LIB.b2_rotate_sum_workspace_bytes(ctx._h, l, n))
    ws, before = torch.empty(nb // 8, dtype=torch.int64, device="cuda"), o.synth_ct(l, 8, 900)
    for first, sum_ in ((1, want), (0, add(want, before, q[:, :l]))):
        acc = dev(before)
        check(LIB.b2_rotate_sum(ctx._h, l, n, e.ctypes.data, src.data_ptr(), 2 * l + 1, tab.ctypes.data, len(tab) // n, acc.data_ptr(), first,
                                ws.data_ptr(), nb, torch.cuda.current_stream().cuda_stream))
        assert np.array_equal(host(acc), sum_)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("log_n,products,sets,dbl", [(12, 16, 1, 0), (14, 3, 2, 1), (16, 1, 2, 1)])
def test_independent_products_in_one_call(log_n, products, sets, dbl):
    """b2_multiply_relin_rescale_many with operands above the level, and b2_rescale_rounded_batch"""
    from pyPhantom._native import LIB, check
    N, l = 1 << log_n, 3
    ctx, o = make_ctx(N, [60, 40, 50, 40, 40, 60, 60], 2)
    key = o.synth_key(o.beta(l), 9, 10)
    rk = ph.relin_key.from_numpy(ctx, key)
    tab, s = rk.pointer_table(), torch.cuda.current_stream().cuda_stream
    la, lb = [l + p % 3 for p in range(products)], [l + (p + 1) % 2 for p in range(products)]
    a = [[o.synth_ct(la[p], 9, 50 + 8 * p + i) for i in range(sets)] for p in range(products)]
    b = [[o.synth_ct(lb[p], 9, 250 + 8 * p + i) for i in range(sets)] for p in range(products)]
    da, db = [dev(np.stack(x)) for x in a], [dev(np.stack(x)) for x in b]
    pa, pb = (np.array([t.data_ptr() for t in d], dtype=np.uint64) for d in (da, db))
    na, nb = np.array(la, dtype=np.uint32), np.array(lb, dtype=np.uint32)
    n_ws = int(LIB.b2_multiply_relin_batch_workspace_bytes(ctx._h, l, products * sets))
    ws = torch.empty(n_ws // 8, dtype=torch.int64, device="cuda")
    out = torch.empty(products, sets, 2, l - 1, N, dtype=torch.int64, device="cuda")
    check(LIB.b2_multiply_relin_rescale_many(ctx._h, l, products, sets, pa.ctypes.data, na.ctypes.data, pb.ctypes.data, nb.ctypes.data, dbl,
                                             tab.ctypes.data, len(tab), out.data_ptr(), ws.data_ptr(), n_ws, s))
    q, got = o.primes[:l][None, :, None], host(out)
    for p in range(products):
        for i in range(sets):
            t = o.tensor_mul(l, a[p][i][:, :l], b[p][i][:, :l])
            t = t * np.uint64(2) % q if dbl else t
            assert np.array_equal(got[p, i], o.rescale_rounded(l, o.keyswitch(l, t[2], key, t[:2]))), (p, i)
    stack = np.stack([o.synth_ct(l, 9, 700 + i) for i in range(sets)])
    res, d = torch.empty(sets, 2, l - 1, N, dtype=torch.int64, device="cuda"), dev(stack)
    check(LIB.b2_rescale_rounded_batch(ctx._h, l, sets, d.data_ptr(), res.data_ptr(), ws.data_ptr(), n_ws, s))
    for i in range(sets):
        assert np.array_equal(host(res)[i], o.rescale_rounded(l, stack[i]))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("l", [1, 8, 9, 16, 17, 24, 25, 32, 33, 48])
def test_composition_at_the_edges_of_its_word_counts(l):
    """b2_decode_compose where the kernel for one more group of eight words takes over: values at 0, Q / 2, Q and between, where
    the quotient's estimate is one off"""
    from pyPhantom._native import LIB, check
    N = 4096
    ctx, o = make_ctx(N, [60, 59] + [40] * 47, 1)
    primes = [int(q) for q in o.primes[:l]]
    Q = int(np.prod(primes, dtype=object))
    rng = np.random.default_rng(l)
    xs = [(k * Q // 16 + d) % Q for k in range(17) for d in (-2, -1, 0, 1, 2)]
    xs += [int.from_bytes(rng.bytes(8 * l), "little") % Q for _ in range(200)] + [int(rng.integers(1 << 62)) % Q for _ in range(50)]
    res = np.zeros((l, N), dtype=np.uint64)
    for k, x in enumerate(xs):
        res[:, k] = [x % q for q in primes]
    d, out = dev(res), torch.empty(N // 2, dtype=torch.complex128, device="cuda")
    check(LIB.b2_decode_compose(ctx._h, l, d.data_ptr(), ph.ckks_encoder(ctx)._crt_table(ctx, l).data_ptr(), 2.0 ** -30, out.data_ptr(),
                                torch.cuda.current_stream().cuda_stream))
    got = torch.view_as_real(out).cpu().numpy()[: len(xs), 0]
    signed = [x - Q if x > Q // 2 else x for x in xs]
    assert np.array_equal(np.sign(got), [(x > 0) - (x < 0) for x in signed])
    small = [k for k, x in enumerate(signed) if abs(x) < 1 << 1000]  # the others are beyond a double
    assert np.allclose(got[small], [float(signed[k]) * 2.0 ** -30 for k in small], rtol=4e-16, atol=0)


@pytest.mark.parametrize("M", [1, 128, 129, 300])
def test_vectors_gathered_from_host_memory(M):
    """b2_gather_vectors at the edges of its table of pointers (128 a launch) and of its rounds of loads"""
    from pyPhantom._native import LIB, check
    N = 4096
    ctx, o = make_ctx(N, [60, 40, 60], 1)
    src = torch.from_numpy(np.random.default_rng(M).integers(-(1 << 62), 1 << 62, (M, N + 2))).pin_memory()
    ptrs = np.array([src.data_ptr() + 8 * (N + 2) * m for m in range(M)], dtype=np.uint64)
    out = torch.zeros(M + 1, N, dtype=torch.int64, device="cuda")
    check(LIB.b2_gather_vectors(ctx._h, M, ptrs.ctypes.data, out.data_ptr(), torch.cuda.current_stream().cuda_stream))
    assert torch.equal(out[:M].cpu(), src[:, :N]) and not out[M].any()


@pytest.mark.parametrize("pool_kb", [400, 800, 1 << 18])
def test_matrix_product_when_the_buffers_come_round(monkeypatch, pool_kb):
    """one, two and four giants a launch; fewer buffers than groups of giants, and enough for all of them"""
    N, l, M, G = 4096, 3, 4, 9
    ctx, o = make_ctx(N, [60, 40, 40, 60], 1, [ph.get_elt_from_step(s, N) for s in (1, 2, 4)])
    keys = {s: o.synth_key(o.beta(l), 3, 10 + 20 * i) for i, s in enumerate((1, 2, 4))}
    glk = ph.galois_key.from_keys([ph.relin_key.from_numpy(ctx, keys[s]) for s in (1, 2, 4)])
    coeffs = [o.synth_signed(5, 70 + d) for d in range(M * G)]
    x_h = o.synth_ct(l, 3, 1)
    x = ph.ciphertext.from_numpy(ctx, x_h, 1, 2.0 ** 40)
    diags = ph.bsgs_diagonals([ph.single_chain_plaintext(c, 2.0 ** 40) for c in coeffs], M * G, M, G)
    monkeypatch.setattr(ph, "_GIANT_POOL_BYTES", pool_kb << 10)
    want = o.bsgs_matmul(l, x_h, coeffs, M, G, keys)
    for _ in range(2):
        assert np.array_equal(ph.bsgs_matmul_preencoded(ctx, glk, x, diags).numpy(), want)


def _matrix_product(M, G, missing=None):
    """a context, its keys (the one of step `missing` left out), a ciphertext, the diagonals' coefficients and the oracle's product"""
    N, l = 4096, 3
    steps = ph.bsgs_required_steps(M)
    ctx, o = make_ctx(N, [60, 40, 40, 60], 1, [ph.get_elt_from_step(s, N) for s in steps])
    keys = {s: o.synth_key(o.beta(l), 3, 10 + 20 * i) for i, s in enumerate(steps)}
    glk = ph.galois_key.from_keys([ph.relin_key() if s == missing else ph.relin_key.from_numpy(ctx, keys[s]) for s in steps])
    coeffs = [o.synth_signed(5, 70 + d) for d in range(M * G)]
    x_h = o.synth_ct(l, 3, 1)
    want = o.bsgs_matmul(l, x_h, coeffs, M, G, keys) if missing is None else None
    return ctx, glk, ph.ciphertext.from_numpy(ctx, x_h, 1, 2.0 ** 40), coeffs, want


def _diagonals(coeffs, M):
    return ph.bsgs_diagonals([ph.single_chain_plaintext(c, 2.0 ** 40) for c in coeffs], len(coeffs), M, len(coeffs) // M)


def test_matrix_products_of_two_streams_do_not_wait_for_one_another():
    """a product behind a stream that is busy for a while; one of another stream is done long before it"""
    ctx, glk, x, coeffs, want = _matrix_product(4, 3)
    diags, streams, got = _diagonals(coeffs, 4), [torch.cuda.Stream() for _ in range(2)], []
    for s in streams:  # what the first calls on a stream set up is there
        with torch.cuda.stream(s):
            ph.bsgs_matmul_preencoded(ctx, glk, x, diags)
    torch.cuda.synchronize()
    for s, busy in zip(streams, (600_000_000, 0)):
        with torch.cuda.stream(s):
            torch.cuda._sleep(busy)
            got.append(ph.bsgs_matmul_preencoded(ctx, glk, x, diags))
    streams[1].synchronize()
    assert not streams[0].query()
    torch.cuda.synchronize()
    for c in got:
        assert np.array_equal(c.numpy(), want)
    sets = []
    for s in streams + [streams[0]]:
        with torch.cuda.stream(s):
            sets.append([t.cuda_stream for t in ctx.product_streams()])
            assert {t.device.index for t in ctx.product_streams()} == {ctx.device}
    assert sets[0] == sets[2] and not set(sets[0]) & set(sets[1])


def test_failed_matrix_product_leaves_no_stream_behind():
    """a baby step without a key is noticed after the first diagonals are on their way: the caller's stream waits for the side
    streams before the call's buffers can be used again"""
    ctx, glk, x, coeffs, _ = _matrix_product(4, 3, missing=2)
    diags = _diagonals(coeffs, 4)
    torch.cuda.synchronize()
    for side in ctx.product_streams()[:3]:
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)
        with pytest.raises(ValueError):
            ph.bsgs_matmul_preencoded(ctx, glk, x, diags)
        assert not torch.cuda.current_stream().query()
        torch.cuda.synchronize()
        assert torch.cuda.current_stream().query()


def test_diagonals_are_read_where_they_are_now():
    """copies of pinned diagonals (their vectors are pageable), a vector that moved since it was set, and vectors in device memory"""
    import copy
    import pickle
    ctx, glk, x, coeffs, want = _matrix_product(4, 3)
    diags = _diagonals(coeffs, 4)
    moved, on_device, mixed = _diagonals(coeffs, 4), _diagonals(coeffs, 4), _diagonals(coeffs, 4)
    for scp in moved.diagonals:
        scp.coeffs.data = scp.coeffs.clone()
    for scp in on_device.diagonals:
        scp.coeffs = scp.coeffs.cuda()
    mixed.diagonals[5] = copy.deepcopy(mixed.diagonals[5])
    for d in (diags, copy.copy(diags), copy.deepcopy(diags), pickle.loads(pickle.dumps(diags)), moved, on_device, mixed):
        assert np.array_equal(ph.bsgs_matmul_preencoded(ctx, glk, x, d).numpy(), want)
    assert diags.diagonals[0].readable_at() == diags.diagonals[0].coeffs.data_ptr()
    assert not any(d.diagonals[0].readable_at() for d in (moved, on_device))


@pytest.mark.parametrize("how", ["deleted", "replaced"])
def test_diagonals_let_go_of_while_a_product_reads_them(how):
    """the reads wait behind a busy stream; the vectors' memory is not handed out again before they are done"""
    ctx, glk, x, coeffs, want = _matrix_product(4, 3)
    diags = _diagonals(coeffs, 4)
    ph.bsgs_matmul_preencoded(ctx, glk, x, diags)
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)
    got = ph.bsgs_matmul_preencoded(ctx, glk, x, diags)
    assert not torch.cuda.current_stream().query()
    if how == "deleted":
        del diags
    else:
        for scp in diags.diagonals:
            scp.coeffs = None
    others = [torch.full((ctx.N,), 1 << 40, dtype=torch.int64).pin_memory() for _ in coeffs]
    assert np.array_equal(got.numpy(), want) and len(others) == len(coeffs)


def test_captured_matrix_product():
    """replays of a captured product; its diagonals are let go of when the graph is"""
    ctx, glk, x, coeffs, want = _matrix_product(4, 3)
    diags = _diagonals(coeffs, 4)
    ph.bsgs_matmul_preencoded(ctx, glk, x, diags)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = ph.bsgs_matmul_preencoded(ctx, glk, x, diags)
    for _ in range(2):
        got.data.zero_()
        graph.replay()
        assert np.array_equal(got.numpy(), want)
    torch.cuda.synchronize()
    del graph
    for scp in diags.diagonals:
        scp.coeffs = None


def test_resident_product_with_keys_loaded_anew_or_cut():
    """a plan uses the digits that its keys hold at the call: loaded anew from other bytes they give what a plan made from those
    gives, and a key cut below the level's digits is refused"""
    import io
    from pyPhantom.linalg import resident_bsgs
    N, l, M, G = 4096, 3, 2, 3
    steps = [1, 2, 4]
    ctx, o = make_ctx(N, [60, 40, 40, 60], 1, [ph.get_elt_from_step(s, N) for s in steps])
    sets = [[ph.relin_key.from_numpy(ctx, o.synth_key(o.beta(l), seed, 10 + 20 * i)) for i in range(3)] for seed in (3, 4)]
    x = ph.ciphertext.from_numpy(ctx, o.synth_ct(l, 3, 1), 1, 2.0 ** 40)
    diags = _diagonals([o.synth_signed(5, 70 + d) for d in range(M * G)], M)
    plan, other = (resident_bsgs(ctx, ph.galois_key.from_keys(keys), diags, 1) for keys in sets)
    before, want = plan.apply(x).numpy(), other.apply(x).numpy()
    assert not np.array_equal(before, want)
    for key, new in zip(*sets):
        buf = io.BytesIO()
        new.save(buf)
        buf.seek(0)
        key.load(buf)
    assert np.array_equal(plan.apply(x).numpy(), want)
    sets[0][1].mod_drop_to_inplace(ctx, 2)
    with pytest.raises(ValueError):
        plan.apply(x)


def test_encoder_checks_the_chain_it_encodes_for():
    """an encoder belongs to a ring; the limits of what fits are those of the context given with the call, longer or shorter"""
    N = 4096
    ctxs = [make_ctx(N, bits, 1)[0] for bits in ([50, 30, 50], [60, 40, 40, 40, 60])]
    values = np.linspace(-1.0, 1.0, N // 2)
    for enc in (ph.ckks_encoder(c) for c in ctxs):
        for ctx in ctxs:
            same = ph.ckks_encoder(ctx).encode_double_vector(ctx, values, 2.0 ** 40)
            assert torch.equal(enc.encode_double_vector(ctx, values, 2.0 ** 40).data, same.data)
        with pytest.raises(ValueError):  # 80 bits of modulus
            enc.encode_double_vector(ctxs[0], values, 2.0 ** 85)
        with pytest.raises(ValueError):  # scale and value together
            enc.encode_double_vector(ctxs[0], 1024.0 * values, 2.0 ** 71)
        with pytest.raises(ValueError):  # 180 bits of modulus, but coefficients of more than 62
            enc.encode_double_vector(ctxs[1], values, 2.0 ** 85)


def test_decoding_of_limbs_that_lie_apart():
    """a plaintext whose limbs are a strided view decodes as its compact copy does, and stays as it is"""
    N = 4096
    ctx, _ = make_ctx(N, [50, 40, 40, 50], 1)
    enc = ph.ckks_encoder(ctx)
    pt = enc.encode_double_vector(ctx, np.linspace(-1.0, 1.0, N // 2), 2.0 ** 40)
    want, limbs = enc.decode_complex_vector(ctx, pt), pt.data
    apart = torch.zeros(5, N, dtype=torch.int64, device="cuda")
    apart[::2] = limbs
    pt.data = apart[::2]
    assert np.array_equal(enc.decode_complex_vector(ctx, pt), want)
    assert torch.equal(apart[::2], limbs) and not apart[1::2].any()


def test_more_vectors_than_a_grid_dimension_holds():
    """b2_expand_single_chain_batch beyond 65535 vectors (4 GB): every one as b2_expand_single_chain makes it"""
    from pyPhantom._native import LIB, check
    N, M, K = 4096, 65537, 7
    ctx, o = make_ctx(N, [40, 40, 60], 1)
    s = torch.cuda.current_stream().cuda_stream
    base = torch.from_numpy(np.stack([o.synth_signed(5, 70 + k) for k in range(K)])).cuda()
    want = ctx.empty(K, 1)
    for k in range(K):
        check(LIB.b2_expand_single_chain(ctx._h, 1, base[k].data_ptr(), want[k].data_ptr(), s))
    src, out = base.repeat(M // K + 1, 1)[:M].contiguous(), ctx.empty(M, 1)
    check(LIB.b2_expand_single_chain_batch(ctx._h, 1, M, src.data_ptr(), out.data_ptr(), s))
    for m in range(0, M, 8192 * K):
        part = out[m: m + 8192 * K, 0]
        assert torch.equal(part, want[:, 0].repeat(8192, 1)[: len(part)])


def test_more_limbs_than_a_grid_dimension_holds():
    """b2_galois_permute beyond 65535 limbs (2 GB each way)"""
    from pyPhantom._native import LIB, check
    N, n = 4096, 65537
    elt = ph.get_elt_from_step(3, N)
    ctx, o = make_ctx(N, [40, 40, 60], 1, [elt])
    src = torch.arange(n * N, dtype=torch.int64, device="cuda").reshape(n, N)
    dst = torch.empty_like(src)
    check(LIB.b2_galois_permute(ctx._h, elt, src.data_ptr(), dst.data_ptr(), n, torch.cuda.current_stream().cuda_stream))
    perm = torch.from_numpy(o.galois_perm(elt).astype(np.int64)).cuda()
    for t in range(0, n, 16384):
        assert torch.equal(dst[t: t + 16384], src[t: t + 16384][:, perm])


@pytest.mark.parametrize("log_n,bits,l", [(12, [60, 40, 50, 60], 3), (13, [40, 50, 36, 30, 60], 4), (14, [50, 40, 30, 45, 60], 4)])
def test_batched_transforms_on_both_sides_of_the_whole_ones(log_n, bits, l):
    """a stack of polynomials transformed in one launch: 192 limbs at 2^12 and 32 at 2^13 and 2^14 are the last that run as whole
    transforms, one polynomial more as two passes"""
    from pyPhantom._native import LIB, check
    N, line = 1 << log_n, 192 if log_n == 12 else 32
    ctx, o = make_ctx(N, bits, 1)
    base = [o.synth_signed(5, 70 + k) for k in range(3)]
    want = torch.stack([dev(o.expand_single_chain(l, b)) for b in base])
    for M in (line // l, line // l + 1):
        src, out = torch.from_numpy(np.stack([base[m % 3] for m in range(M)])).cuda(), ctx.empty(M, l)
        check(LIB.b2_expand_single_chain_batch(ctx._h, l, M, src.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream))
        assert torch.equal(out, want[torch.arange(M, device="cuda") % 3])


@pytest.mark.parametrize("batch", [1, 6, 7, 12, 13, 25])
def test_key_switches_on_both_sides_of_the_whole_conversions(batch):
    """2^12 with eight special primes: ModUp's 8 limbs a set and ModDown's 16 are converted while they load up to 96 a launch,
    the inverse transforms' 8 run whole up to 192; every set of a batch as it is alone, the first and last as the oracle has
    them, and so for hoisted and for summed rotations"""
    from pyPhantom._native import LIB, check
    N, l, n_elt = 4096, 8, 2
    elts = [ph.get_elt_from_step(s, N) for s in (1, 2)]
    ctx, o = make_ctx(N, [60] + [40, 50, 36, 40, 45, 40, 40] + [60] * 7 + [59], 8, elts)
    key = o.synth_key(o.beta(l), 4, 10)
    a, b = ([o.synth_ct(l, 4, at + i) for i in range(batch)] for at in (20, 60))
    da, db, rk = dev(np.stack(a)), dev(np.stack(b)), _key(ctx, key)
    got = ph.multiply_relin_rescale_batch(ctx, da, db, rk)
    for i in range(batch):
        assert torch.equal(got[i], ph.multiply_relin_rescale_batch(ctx, da[i: i + 1], db[i: i + 1], rk)[0])
    for i in {0, batch - 1}:
        assert np.array_equal(host(got[i]), o.rescale(l, o.multiply_and_relin(l, a[i], b[i], key)))
    keys = [o.synth_key(o.beta(l), 6, 100 + 40 * i) for i in range(n_elt)]
    rks = [_key(ctx, k) for k in keys]
    glk, ct = ph.galois_key.from_keys(rks), ph.ciphertext.from_numpy(ctx, a[0], 1)
    steps = [1 + i % 2 for i in range(batch)]
    want = o.hoist_rotations(l, a[0], elts, keys)
    for i, c in enumerate(ph.hoist_rotations(ctx, ct, glk, steps)):
        assert np.array_equal(c.numpy(), want[i % 2])
    tab = np.concatenate([rks[i % 2].pointer_table() for i in range(batch)])
    e, nb = np.array([elts[i % 2] for i in range(batch)], dtype=np.uint32), int(LIB.b2_rotate_sum_workspace_bytes(ctx._h, l, batch))
    ws, acc = torch.empty(nb // 8, dtype=torch.int64, device="cuda"), ctx.empty(2, l)
    check(LIB.b2_rotate_sum(ctx._h, l, batch, e.ctypes.data, da.data_ptr(), 2 * l, tab.ctypes.data, o.beta(l), acc.data_ptr(), 1, ws.data_ptr(), nb,
                            torch.cuda.current_stream().cuda_stream))
    q = np.concatenate([o.primes[:l], o.primes[-8:]])[None, :, None]
    cx, c0 = 0, 0
    for i in range(batch):
        turned = a[i][:, :, o.galois_perm(elts[i % 2])]
        cx = (o.ks_inner_prod(l, o.modup(l, turned[1]), keys[i % 2]) + cx) % q
        c0 = (turned[0] + c0) % q[0, :l]
    want = np.stack([o.moddown(l, cx[k]) for k in range(2)])
    want[0] = (want[0] + c0) % q[0, :l]
    assert np.array_equal(host(acc), want)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("sets", [32, 33])
def test_rescales_on_both_sides_of_the_whole_ones(sets):
    """2^12: six limbs a ciphertext, whole up to 192 a launch"""
    from pyPhantom._native import LIB, check
    N, l = 4096, 4
    ctx, o = make_ctx(N, [60, 40, 50, 45, 60], 1)
    cts = [o.synth_ct(l, 9, 700 + i) for i in range(sets)]
    d, res, ws = dev(np.stack(cts)), torch.empty(sets, 2, l - 1, N, dtype=torch.int64, device="cuda"), ctx.empty(2 * sets)
    check(LIB.b2_rescale_rounded_batch(ctx._h, l, sets, d.data_ptr(), res.data_ptr(), ws.data_ptr(), ws.numel() * 8, torch.cuda.current_stream().cuda_stream))
    got = host(res)
    for i in range(sets):
        assert np.array_equal(got[i], o.rescale_rounded(l, cts[i]))


@pytest.mark.parametrize("log_n", [13, 14])
@pytest.mark.parametrize("first,n", [(1, 1), (1, 32), (1, 33), (0, 1), (0, 5), (30, 5)])
def test_transforms_of_ranges_of_limbs(log_n, first, n):
    """forward and inverse, on FP64 primes alone (whole transforms up to 32 limbs) and with a 60-bit one at either end"""
    from pyPhantom._native import LIB, check
    N = 1 << log_n
    ctx, o = make_ctx(N, [60] + [40, 50, 36] * 11 + [60], 1)
    x = o.fill(1, o.primes[first: first + n], 9, 50)[0]
    for call, want in ((LIB.b2_ntt_forward, o.ntt_forward(x, first)), (LIB.b2_ntt_inverse, o.ntt_inverse(x, first))):
        d = dev(x)
        check(call(ctx._h, d.data_ptr(), n, first, torch.cuda.current_stream().cuda_stream))
        assert np.array_equal(host(d), want)


@pytest.mark.parametrize("log_n,special,l,below", [
    (15, 2, 6, 15),   # three digits: four and a half waves of the fused pass
    (15, 1, 4, 8),    # four digits: one and a half
    (15, 3, 6, 21),   # two digits: seven
    (16, 2, 5, 8),    # a ragged third digit
    (16, 2, 2, 6),    # one digit: never fused
])
def test_batches_on_both_sides_of_the_fused_row_pass(log_n, special, l, below):
    """products with the last batch that stores the row pass on 148 SMs and the first that fuses it (which of the two ran is read
    from the launches): every set as it is alone, the first as the oracle has it"""
    N = 1 << log_n
    ctx, o = make_ctx(N, [60, 40, 50, 36, 40, 45][:l] + [60] * (special - 1) + [59], special)
    key = o.synth_key(o.beta(l), 4, 10)
    rk, a, b = _key(ctx, key), o.synth_ct(l, 4, 20), o.synth_ct(l, 4, 40)
    da, db = (torch.stack([dev(x)] + [dev(o.synth_ct(l, 4, at + i)) for i in range(1, 3)]) for x, at in ((a, 60), (b, 80)))
    one = torch.stack([ph.multiply_relin_rescale_batch(ctx, da[i: i + 1], db[i: i + 1], rk)[0] for i in range(3)])
    assert np.array_equal(host(one[0]), o.rescale(l, o.multiply_and_relin(l, a, b, key)))
    for batch in (below, below + 1):
        pick = torch.arange(batch, device="cuda") % 3
        got, kernels = kernels_of(ctx, lambda: ph.multiply_relin_rescale_batch(ctx, da[pick], db[pick], rk))
        fused = batch > below and o.beta(l) > 1
        assert ("ntt_fwd_rows_mac" in kernels, "ks_inner_prod" in kernels) == (fused, not fused), kernels
        assert torch.equal(got, one[pick])
    assert ctx.device_status() == 0


@pytest.mark.parametrize("log_n,bits,special,l,batch,fused", [
    (13, [60, 40, 50, 36, 45, 30, 60, 60, 60], 3, 6, 1, False),                   # every prime class, full digits
    (13, [60, 40, 46, 36, 50, 45, 40, 60, 59, 60, 60, 60], 5, 7, 2, False),       # five input limbs, then two
    (13, [60] + [40, 50] * 4 + [60] * 8, 8, 9, 2, False),                         # eight input limbs, then one
    (13, [60, 40, 40, 40, 60], 1, 4, 1, False),                                   # one input limb
    (14, [60, 40, 50, 36, 60, 60], 2, 3, 1, False),
    (14, [60, 40, 50, 36, 60, 60], 2, 4, 3, False),
    (14, [60, 40, 50, 36, 40, 60, 60, 60], 3, 5, 1, False),
    (15, [60, 40, 50, 36, 60, 60], 2, 4, 1, False),
    (15, [60, 40, 50, 36, 40, 60, 60], 2, 5, 12, False),
    (15, [60, 40, 50, 36, 40, 60, 60], 2, 5, 18, True),                           # behind it the row pass with the inner product
    (16, [60, 40, 50, 36, 60, 60], 2, 4, 1, True),                                # the same for the FP64 limbs of a single call
    (16, [60, 40, 36, 60, 60], 2, 3, 4, False),
    (16, [60, 40, 50, 36, 40, 60, 60], 2, 5, 9, True),                            # a ragged third digit
])
def test_conversion_in_the_column_pass_equals_the_oracle(log_n, bits, special, l, batch, fused):
    """key switches whose base conversions are made while the forward transforms load, ModUp and ModDown, single and batched (that
    no conversion kernel ran, and which row pass did, is read from the launches)"""
    ctx, o = make_ctx(1 << log_n, bits, special)
    key = o.synth_key(o.beta(l), 8, 10)
    a, b = [o.synth_ct(l, 8, 20 + i) for i in range(batch)], [o.synth_ct(l, 8, 40 + i) for i in range(batch)]
    rlk = _key(ctx, key)
    if batch == 1:
        ca, cb = (ph.ciphertext.from_numpy(ctx, v[0], ctx.size_Q - l + 1, 2.0 ** 40) for v in (a, b))
        res, kernels = kernels_of(ctx, lambda: ph.multiply_and_relin(ctx, ca, cb, rlk))
        got = [host(res.data)]
    else:
        ext = dev(np.stack([o.tensor_mul(l, a[i], b[i]) for i in range(batch)]))
        res, kernels = kernels_of(ctx, lambda: ph.relinearize_batch(ctx, ext, rlk))
        got = host(res)
    assert "bconv" not in kernels and ("ntt_fwd_rows_mac" in kernels) == fused, kernels
    for i in range(batch):
        assert np.array_equal(got[i], o.multiply_and_relin(l, a[i], b[i], key)), f"set {i}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("log_n,special,l,batch", [(12, 7, 8, 7), (13, 1, 5, 0), (14, 4, 9, 3), (14, 5, 5, 3), (14, 3, 27, 3), (15, 8, 17, 3),
                                                   (16, 6, 7, 3), (17, 3, 4, 3)])
def test_pair_conversion_edges(log_n, special, l, batch):
    """the tensor-core conversion at odd numbers of input limbs, ragged digits and column groups that leave its items uneven:
    ModUp (with the digits' own limbs copied) and a batch of key switches, every byte count of an output prime among them; nine
    digits are more jobs than a launch carries in its parameters. Key switches with one input limb run no conversion kernel."""
    from pyPhantom import _native
    from pyPhantom._native import LIB, check
    from gpu_helpers import stream
    bits = ([60, 30, 40, 46, 50, 55, 36, 42] * 4)[:l] + [60] * special
    ctx, o = make_ctx(1 << log_n, bits, special)
    c2 = o.fill(1, o.primes[:l], 3, 7)[0]
    up = ctx.empty(o.beta(l), l + special)
    nb = LIB.b2_workspace_bytes(ctx._h, _native.OP_MODUP, l)
    ws = torch.empty(nb // 8, dtype=torch.int64, device="cuda")
    check(LIB.b2_modup(ctx._h, l, dev(c2).data_ptr(), up.data_ptr(), ws.data_ptr(), nb, stream()))
    want = o.modup(l, c2)
    assert np.array_equal(host(up).reshape(want.shape), want)
    assert ctx.device_status() == 0
    if not batch:
        return
    key = o.synth_key(o.beta(l), 3, 10)
    sets = [o.fill(3, o.primes[:l], 3, 20 + i) for i in range(batch)]
    got, kernels = kernels_of(ctx, lambda: ph.relinearize_batch(ctx, dev(np.stack(sets)), _key(ctx, key)))
    assert kernels["bconv"] == 2, kernels  # ModUp's and ModDown's
    for i, s in enumerate(sets):
        assert np.array_equal(host(got[i]), o.keyswitch(l, s[2], key, s[:2])), f"set {i}"
    assert ctx.device_status() == 0


@pytest.mark.parametrize("log_n,bits,special,l,batch", [
    (12, [60, 40, 40, 30, 60], 1, 4, 1),                          # whole transforms; a short prime goes
    (12, [60, 40, 50, 36, 60, 60, 60], 2, 4, 40),                 # more limbs than whole transforms take
    (13, [60, 40, 40, 60, 60, 60], 2, 4, 1),                      # a 60-bit prime goes; converted in the column pass
    (13, [60, 40, 46, 36, 50] + [60] * 5, 5, 5, 3),
    (14, [60, 40, 36, 45, 40, 50] + [60] * 4, 4, 6, 1),           # converted on the tensor cores
    (14, [60, 40, 36, 45, 40, 50] + [60] * 4, 4, 2, 2),           # one limb is left
    (16, [60, 40, 36, 45, 40] + [60] * 3, 3, 5, 1),
    (16, [60, 40, 36, 45, 40] + [60] * 4, 4, 5, 2),
])
def test_moddown_and_rescale_in_one_equal_the_oracle(log_n, bits, special, l, batch):
    """products relinearised and rescaled by floor (b2_multiply_relin_rescale_batch) and to nearest (.._many), single and batched"""
    from pyPhantom._native import LIB, check
    from gpu_helpers import key_dev, stream
    ctx, o = make_ctx(1 << log_n, bits, special)
    key = o.synth_key(o.beta(l), 6, 10)
    a, b = [o.synth_ct(l, 6, 20 + i) for i in range(batch)], [o.synth_ct(l, 6, 120 + i) for i in range(batch)]
    da, db = dev(np.stack(a)), dev(np.stack(b))
    got = host(ph.multiply_relin_rescale_batch(ctx, da, db, _key(ctx, key)))
    kt, kp = key_dev(key)
    nb = LIB.b2_multiply_relin_batch_workspace_bytes(ctx._h, l, batch)
    ws, out = torch.empty(nb // 8, dtype=torch.int64, device="cuda"), ctx.empty(batch, 2, l - 1)
    pa, pb = (np.array([t.data_ptr()], dtype=np.uint64) for t in (da, db))
    ll = np.array([l], dtype=np.uint32)
    check(LIB.b2_multiply_relin_rescale_many(ctx._h, l, 1, batch, pa.ctypes.data, ll.ctypes.data, pb.ctypes.data, ll.ctypes.data, 0, kp.ctypes.data, len(kp),
                                             out.data_ptr(), ws.data_ptr(), nb, stream()))
    near = host(out)
    for i in range(min(batch, 3)):
        prod = o.multiply_and_relin(l, a[i], b[i], key)
        assert np.array_equal(got[i], o.rescale(l, prod)), f"floor, pair {i}"
        assert np.array_equal(near[i], o.rescale_rounded(l, prod)), f"nearest, pair {i}"
    assert ctx.device_status() == 0
