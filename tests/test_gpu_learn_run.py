"""Launch lists of the learned stop (ems_learn_run): the GEMM with its sum over
k in one chain, operands read along either index, rows of a convolution read in
place, bias and activation in the epilogue; the
activation adjoint with its bias gradient; the loss. Against numpy in f64 on
the bf16-rounded operands.

Bounds: a GEMM's products are exact in f32 and its f32 sums of K terms differ
from f64's by at most K·2^-24·Σ|a·b| <= K·2^-24·|A||B|; the tests allow
4·sqrt(K)·2^-24 of the largest row-column norm product (rounding errors are
independent), and one bf16 rounding (2^-8) for bf16 outputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bf16(x):
    from oracle.cnn import bf16

    r = bf16(np.asarray(x, dtype=np.float32)).astype(np.float32)
    return (r.view(np.uint32) >> 16).astype(np.uint16).view(np.int16), r.astype(np.float64)


def _from_bf16(t):
    return (t.cpu().numpy().view(np.uint16).astype(np.uint32) << 16).view(np.float32).astype(np.float64)


def _run(net, *cmds):
    from ems_b200 import learn as L

    net._run((L.Cmd * len(cmds))(*cmds))
    net.torch.cuda.synchronize()
    assert net.lib.ems_learn_check() == 0


@pytest.fixture(scope="module")
def net():
    from ems_b200 import learn as L

    return L.Net(seed=0)


@pytest.mark.parametrize("M,N,K", [(32, 16, 32704), (64, 64, 3840), (128, 512, 1920), (8, 136, 129), (1, 24, 700),
                                   (130, 16, 128), (257, 40, 65)])
@pytest.mark.parametrize("along", ["k", "rows"])
@pytest.mark.parametrize("bias", [False, True])
def test_split_gemm(net, M, N, K, along, bias):
    t = net.torch
    rng = np.random.default_rng(M + 3 * N + 7 * K)
    (ab, a), (bb, b) = (_bf16(rng.standard_normal(s)) for s in ((M, K), (K, N)))
    if along == "rows":  # A(i, k) and B(k, j) contiguous along i and j
        A, sa = t.from_numpy(np.ascontiguousarray(ab.T)).cuda(), (1, M)
        B, sb = t.from_numpy(bb).cuda(), (N, 1)
    else:
        A, sa = t.from_numpy(ab).cuda(), (K, 1)
        B, sb = t.from_numpy(np.ascontiguousarray(bb.T)).cuda(), (1, K)
    v = rng.standard_normal(N).astype(np.float32)
    C, F = (t.empty(M, N, device="cuda") for _ in range(2))
    H = t.empty(M, N, dtype=t.int16, device="cuda")
    want = a @ b
    tol = 4 * np.sqrt(K) * 2.0 ** -24 * np.max(np.linalg.norm(a, axis=1)) * np.max(np.linalg.norm(b, axis=0))
    if bias:
        V = t.from_numpy(v).cuda()
        _run(net, net._gemm(A, sa, B, sb, M, N, K, C, bias=V, act=1, outb=H, outf=F))
        want = want + v
        silu = want / (1 + np.exp(-want))
        # |silu'| <= 1.1; 4 ulp of f32 for the activation itself.
        assert np.max(np.abs(F.cpu().numpy() - silu) - 2.0 ** -21 * np.abs(silu)) <= 1.1 * tol
        assert np.max(np.abs(_from_bf16(H) - silu) - 2.0 ** -8 * np.abs(silu)) <= 1.1 * tol
    else:
        _run(net, net._gemm(A, sa, B, sb, M, N, K, C))
    assert np.max(np.abs(C.cpu().numpy() - want) - 2.0 ** -23 * np.abs(want)) <= tol


@pytest.mark.parametrize("B,T,C,k,s,N", [(3, 61, 8, 8, 4, 32), (2, 40, 2, 8, 4, 16), (5, 19, 3, 5, 2, 9)])
def test_convolution_rows_in_place(net, B, T, C, k, s, N):
    """Forward rows (two-level row index of A) and the weight gradient's (of
    B's k index); the last shape allows no vector reads."""
    t = net.torch
    rng = np.random.default_rng(T)
    To = (T - k) // s + 1
    xb, x = _bf16(rng.standard_normal((B, T, C)))
    wb, w = _bf16(rng.standard_normal((N, k * C)))
    db, d = _bf16(rng.standard_normal((B * To, N)))
    X, Wt, D = (t.from_numpy(v).cuda() for v in (xb, wb, db))
    Y = t.empty(B * To, N, device="cuda")
    G = t.empty(N, k * C, device="cuda")
    _run(net, net._gemm(X, (s * C, 1), Wt, (1, k * C), B * To, N, k * C, Y, rows_a=(To, T * C)),
         net._gemm(D, (1, N), X, (s * C, 1), N, k * C, B * To, G, rows_b=(To, T * C)))
    cols = np.stack([x[q, r * s:r * s + k].ravel() for q in range(B) for r in range(To)])
    for got, want, n in ((Y, cols @ w.T, k * C), (G, d.T @ cols, B * To)):
        assert np.max(np.abs(got.cpu().numpy() - want)) <= 4 * np.sqrt(n) * 2.0 ** -24 * n * 12


@pytest.mark.parametrize("B,T,cols,k,s", [(2, 19, 32, 8, 4), (3, 23, 3, 5, 2), (1, 7, 300, 3, 3)])
@pytest.mark.parametrize("act", [0, 1])
def test_activation_adjoint(net, B, T, cols, k, s, act):
    from oracle.cnn import col2im, silu_grad

    t = net.torch
    rng = np.random.default_rng(T + act)
    To = (T - k) // s + 1
    d = rng.standard_normal((B * To, k * cols)).astype(np.float32)
    y = rng.standard_normal((B * T, cols)).astype(np.float32)
    da = col2im(d.astype(np.float64), B, T, cols, k, s).reshape(B * T, cols)
    want = da * (silu_grad(y.astype(np.float64)) if act else 1.0)
    D, Y = t.from_numpy(d).cuda(), t.from_numpy(y).cuda()
    for conv, src in (((T, k, s), D), (None, t.from_numpy(da.astype(np.float32)).cuda())):
        H = t.empty(B * T, cols, dtype=t.int16, device="cuda")
        S = t.empty(cols, device="cuda")
        _run(net, net._dy(Y, src, H, S, B * T, cols, act, conv))
        scale = np.max(np.abs(want))
        assert np.max(np.abs(_from_bf16(H) - want) - 2.0 ** -8 * np.abs(want)) <= 2.0 ** -20 * scale
        assert np.max(np.abs(S.cpu().numpy() - want.sum(axis=0))) <= B * T * 2.0 ** -20 * scale


@pytest.mark.parametrize("n", [1, 255, 49152, 100001])
def test_loss(net, n):
    from ems_b200 import learn as L

    t = net.torch
    rng = np.random.default_rng(n)
    a, b = rng.standard_normal((2, n)).astype(np.float32)
    A, Bt = t.from_numpy(a).cuda(), t.from_numpy(b).cuda()
    G, loss, sh = t.empty(n, device="cuda"), t.empty(1, device="cuda"), t.empty(64, device="cuda")
    _run(net, net._cmd(L.MSE, s=(n,), p=(A, Bt, G, loss, sh)))
    d = a.astype(np.float64) - b
    assert abs(float(loss.item()) - np.mean(d * d)) <= 1e-6 * np.mean(d * d)
    np.testing.assert_allclose(G.cpu().numpy(), 2 * d / n, rtol=1e-6, atol=2.0 ** -23 * 8 / n)


@pytest.mark.parametrize("B", [1, 3, 70])
def test_network_at_other_batch_sizes(B):
    from ems_b200 import learn as L
    from oracle import cnn

    net = L.Net(seed=2)
    t = net.torch
    rng = np.random.default_rng(B)
    for b in (B, B + 1):  # the lists are built again for another size
        x = rng.standard_normal((b, L.K_IN, 2)).astype(np.float32)
        dout = rng.standard_normal((b, 2 * L.T_OUT)).astype(np.float32)
        out = net.forward(t.from_numpy(x).cuda()).cpu().numpy()
        net.backward(t.from_numpy(dout).cuda())
        want, cache = cnn.forward(L.init_params(2), x, L.T_OUT)
        assert np.linalg.norm(out - want) <= 5e-3 * np.linalg.norm(want)
        g = cnn.backward(cache, dout, L.T_OUT)
        assert np.linalg.norm(net.g.cpu().numpy() - g) <= 2e-2 * np.linalg.norm(g)


def _bits(t):
    return t.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("B", [2, 33, 130])
def test_rows_of_a_batch_come_out_as_alone(B):
    """Every output is one sum over k in order, whatever the batch: bit for bit."""
    from ems_b200 import learn as L

    net = L.Net(seed=4)
    x = net.torch.from_numpy(np.random.default_rng(B).standard_normal((B, L.K_IN, 2)).astype(np.float32)).cuda()
    out = _bits(net.forward(x))
    for q in (0, B // 2, B - 1):
        assert np.array_equal(_bits(net.forward(x[q:q + 1]))[0], out[q]), q


@pytest.mark.parametrize("rows,cols", [(1, 1), (255, 3), (256, 4), (257, 32), (5000, 5), (32704, 32), (64, 768)])
def test_bias_gradient_is_summed_as_bias_grad(net, rows, cols):
    t = net.torch
    d = t.from_numpy(np.random.default_rng(rows).standard_normal((rows, cols)).astype(np.float32)).cuda()
    H, S, want = t.empty(rows, cols, dtype=t.int16, device="cuda"), t.empty(cols, device="cuda"), t.empty(cols, device="cuda")
    _run(net, net._dy(None, d, H, S, rows, cols, 0))
    assert net.lib.ems_learn_bias_grad(net._ptr(d), net._ptr(want), rows, cols, net._s()) == 0
    assert np.array_equal(_bits(S), _bits(want))


def test_bias_gradients_put_off_to_the_end_of_the_list(net):
    """Eight of them: six in one launch, two in the next; uneven matrices."""
    t = net.torch
    rng = np.random.default_rng(3)
    shapes = [(1, 1), (300, 33), (64, 768), (4097, 64), (255, 8), (256, 31), (1000, 7), (513, 129)]
    d = [t.from_numpy(rng.standard_normal(s).astype(np.float32)).cuda() for s in shapes]
    S = [t.empty(s[1], device="cuda") for s in shapes]
    H = [t.empty(s, dtype=t.int16, device="cuda") for s in shapes]
    _run(net, *[net._dy(None, d[q], H[q], S[q], *shapes[q], 0, later=True) for q in range(8)])
    for q, (rows, cols) in enumerate(shapes):
        want = t.empty(cols, device="cuda")
        assert net.lib.ems_learn_bias_grad(net._ptr(d[q]), net._ptr(want), rows, cols, net._s()) == 0
        assert np.array_equal(_bits(S[q]), _bits(want)), (rows, cols)


@pytest.mark.parametrize("n", [1, 1025, 49152, 100001])
def test_loss_is_summed_as_mse(net, n):
    from ems_b200 import learn as L

    t = net.torch
    a, b = (t.from_numpy(v).cuda() for v in np.random.default_rng(n).standard_normal((2, n)).astype(np.float32))
    G, loss, sh, G1, want = (t.empty(q, device="cuda") for q in (n, 1, 64, n, 1))
    _run(net, net._cmd(L.MSE, s=(n,), p=(a, b, G, loss, sh)))
    assert net.lib.ems_learn_mse(net._ptr(a), net._ptr(b), net._ptr(G1), net._ptr(want), n, net._s()) == 0
    assert np.array_equal(_bits(G), _bits(G1)) and np.array_equal(_bits(loss), _bits(want))


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (15, 17, 15), (16, 16, 16), (17, 15, 17), (127, 129, 63), (128, 128, 64),
                                   (129, 127, 65), (24, 40, 255), (40, 24, 256), (8, 8, 257), (32, 16, 2047),
                                   (128, 64, 769), (256, 256, 320)])
def test_layouts_and_joined_launches_agree(net, M, N, K):
    """Operands read along k, along the rows and element by element (tiles',
    stages' and vectors' edges), alone and several in a launch: the same bits,
    and the value within the bound above."""
    t = net.torch
    rng = np.random.default_rng(M + N + K)
    (ab, a), (bb, b) = (_bf16(rng.standard_normal(s)) for s in ((M, K), (K, N)))
    up = lambda n: (n + 7) // 8 * 8  # noqa: E731

    def lay(v, ld, off=0):  # rows of v `ld` elements apart, from element `off` of an allocation on
        buf = t.zeros(off + v.shape[0] * ld, dtype=t.int16, device="cuda")
        buf[off:].view(v.shape[0], ld)[:, :v.shape[1]] = t.from_numpy(np.ascontiguousarray(v)).cuda()
        return buf[off:]

    A = [(lay(ab, up(K)), (up(K), 1)), (lay(ab.T, up(M)), (1, up(M))), (lay(ab, K + 1, 1), (K + 1, 1))]
    Bs = [(lay(bb.T, up(K)), (1, up(K))), (lay(bb, up(N)), (up(N), 1)), (lay(bb, N + 1, 1), (N + 1, 1))]
    C = [t.empty(M, N, device="cuda") for _ in range(9)]
    cmds = [net._gemm(*A[q % 3], *Bs[q // 3], M, N, K, C[q]) for q in range(9)]
    for c in cmds:
        _run(net, c)
    one = [_bits(c) for c in C]
    tol = 4 * np.sqrt(K) * 2.0 ** -24 * np.max(np.linalg.norm(a, axis=1)) * np.max(np.linalg.norm(b, axis=0))
    assert np.max(np.abs(C[0].cpu().numpy() - a @ b)) <= tol + 2.0 ** -23 * np.max(np.abs(a @ b))
    for q in range(1, 9):
        assert np.array_equal(one[q], one[0]), q
    for q, c in enumerate(cmds):
        C[q].zero_()
        c.i[6] = int(q > 0)
    _run(net, *cmds)  # six products in the first launch, three in the second
    for q in range(9):
        assert np.array_equal(_bits(C[q]), one[0]), q


def test_backward_takes_gradients_of_other_types_and_places():
    from ems_b200 import learn as L

    net = L.Net(seed=5)
    t = net.torch
    rng = np.random.default_rng(1)
    net.forward(t.from_numpy(rng.standard_normal((5, L.K_IN, 2)).astype(np.float32)).cuda())
    d = t.from_numpy(rng.standard_normal((5, 2 * L.T_OUT)).astype(np.float32)).cuda()
    net.backward(d)
    want = _bits(net.g)
    for other in (d.cpu(), d.double(), d.t().contiguous().t()):
        net.g.zero_()
        net.backward(other)
        assert np.array_equal(_bits(net.g), want)
    for bad in (d[:4], d[:, :-1], t.cat([d, d])):
        with pytest.raises(RuntimeError):
            net.backward(bad)
    net.train_step(t.zeros(3, L.K_IN, 2, device="cuda"), t.zeros(3, 2 * L.T_OUT, device="cuda"))
