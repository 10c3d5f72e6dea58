"""Tile edges of the surrogate's kernels on the GPU: narrow and wide GEMM tiles
with ragged last tiles, and whole training steps (loss gradient in the output
GEMM, split weight gradients, bias sums) of odd shapes, one layer to seven.
"""
import ctypes as C
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


# 128-row tiles of 32 columns up to 148 of them, then 64, then 128; 256 for many tiles of long sums
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 512, 512), (129, 40, 72), (127, 232, 320), (18 * 128, 24, 64),
                                   (18 * 128 + 1, 24, 64), (9 * 128, 264, 136), (9 * 128 + 2, 264, 136),
                                   (37 * 128, 128, 64), (37 * 128 + 1, 128, 64),  # 148 tiles of 32, 149 of 32
                                   (1283, 504, 200), (37 * 128, 256, 8), (37 * 128 + 5, 256, 8),  # 64, and past it
                                   (2435, 1000, 72), (37 * 128, 1024, 1024), (5119, 1000, 1032)])  # 128, 128, 256
def test_gemm_tile_edges(lcb, M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    A = torch.randn(M, K, device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn(N, K, device="cuda", generator=g).to(torch.bfloat16)
    bias, aux = torch.randn(N, device="cuda", generator=g), torch.randn(M, N, device="cuda", generator=g)
    ref = A.double() @ B.double().T
    # FP32 accumulation of K exact products, K + 1 roundings of at most 2^-24 of the sum of |terms|
    # each, doubled for the pairwise order the tensor cores are free to use
    bound = (K + 2) * 2.0 ** -23 * (A.double().abs() @ B.double().abs().T + bias.double().abs())
    L = lcb._capi.load()
    for mode in range(4):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32 if mode in (0, 2) else torch.bfloat16)
        z = torch.empty(M, N, device="cuda")
        err = torch.zeros(1, device="cuda", dtype=torch.int32)
        lcb._capi.check_mlp(L.lcb_mlp_gemm(mode, M, N, K, _ptr(A), _ptr(B), _ptr(bias), _ptr(aux), _ptr(out), _ptr(z),
                                           _ptr(err), None))
        torch.cuda.synchronize()
        assert int(err.item()) == 0
        if mode == 0:
            want, tol = ref, bound
        elif mode == 2:
            want, tol = ref + bias.double(), bound
        elif mode == 1:  # GELU has a slope below 1.13; BF16 rounding 2^-8 of the value; 1e-6 for erff's ulps
            want = torch.nn.functional.gelu(ref + bias.double())
            tol = 1.13 * bound + 2.0 ** -8 * want.abs() + 1e-6
            assert bool(((z.double() - (ref + bias.double())).abs() <= bound).all())
        else:
            x = aux.double().requires_grad_(True)
            torch.nn.functional.gelu(x).sum().backward()
            want = ref * x.grad
            tol = bound * 1.13 + 2.0 ** -8 * want.abs() + 1e-6 * (1 + ref.abs())
        assert bool(((out.double() - want).abs() <= tol).all()), mode


@pytest.mark.parametrize("B,n_in,width,hidden,n_out,skew", [(8, 1, 8, 1, 8, 0), (200, 5, 40, 2, 24, 1), (136, 9, 264, 1, 264, 0),
                                                            (1032, 5, 136, 3, 40, 1), (64, 3, 24, 7, 16, 0)])
def test_training_step_shapes(lcb, B, n_in, width, hidden, n_out, skew):
    from oracle import mlp_oracle as MO

    shape = dict(n_in=n_in, width=width, n_hidden=hidden, n_out=n_out)
    L = lcb._capi.load()
    h = C.c_void_p()
    lcb._capi.check_mlp(L.lcb_mlp_create(0, n_in, width, hidden, n_out, B, 7, C.byref(h)))
    try:
        n = C.c_int64()
        lcb._capi.check_mlp(L.lcb_mlp_num_params(h, C.byref(n)))
        rng = np.random.default_rng(B)
        x = rng.uniform(-1, 1, (B, n_in)).astype(np.float32)
        t = rng.normal(0, 1, (B, n_out)).astype(np.float32)
        params, grads = np.empty(n.value, np.float32), np.empty(n.value, np.float32)
        lcb._capi.check_mlp(L.lcb_mlp_get_params(h, params.ctypes.data, n.value))
        xd = torch.from_numpy(x).cuda()
        td = torch.empty(B * n_out + skew, device="cuda")[skew:]  # targets off a 16-byte boundary too
        td.copy_(torch.from_numpy(t.ravel()))
        torch.cuda.synchronize()  # the network works on its own stream
        for _ in range(2):  # the second pass overwrites the first one's gradients
            lcb._capi.check_mlp(L.lcb_mlp_backward(h, _ptr(xd), _ptr(td), B))
        lcb._capi.check_mlp(L.lcb_mlp_get_grads(h, grads.ctypes.data, n.value))
        loss = C.c_double()
        lcb._capi.check_mlp(L.lcb_mlp_take_loss(h, C.byref(loss)))
        want_loss, want, _ = MO.loss_and_grads(params.astype(np.float64), x, t, **shape)
        assert abs(loss.value - 2 * want_loss) <= 2e-3 * want_loss
        # BF16 gradients between layers: a flip of one ulp (2^-8) of a few of them stays below 1e-2 of the norm
        k, sizes = 0, []
        for i in range(hidden + 1):
            o, fan = (n_out if i == hidden else width), (n_in if i == 0 else width)
            sizes += [o * fan, o]
        assert sum(sizes) == n.value
        for size in sizes:
            g, r = grads[k:k + size], want[k:k + size]
            assert np.linalg.norm(g - r) <= 1e-2 * np.linalg.norm(r) + 1e-12, (k, size)
            k += size
    finally:
        L.lcb_mlp_destroy(h)


@pytest.mark.parametrize("walkers,moves", [(1, 1), (33, 2), (130, 3)])
def test_subchain_rows(lcb, walkers, moves):
    """The packed input rows and the fused accept step at few and ragged rows, against the host loop."""
    S, M = importlib.import_module("lcurve-rs_b200.surrogate"), importlib.import_module("lcurve-rs_b200.mcmc")
    W = importlib.import_module("lcurve-rs_b200.workloads")
    setup = S.CurveSetup()
    flux = np.linspace(1.0, 1.1, len(setup.times))
    sur = S.Surrogate(seed=4)
    sur.bind_data(W.noisy_data(setup.times, flux, setup.expose, setup.ndiv, seed=1))
    both = M.initial_walkers(2 * max(walkers, 16), S.TRUTH, seed=2, spread=0.05)
    y, comp = both[:walkers], both[walkers:]
    ls = -0.5 * sur.chisq(y)
    for move in ("stretch", "kde"):
        rnd = M.subchain_numbers(np.random.default_rng(5), moves, walkers, move)
        yd, lsd = sur.subchain(y, ls, comp, rnd, move=move)
        yh, lsh = M.subchain_host(sur, y, ls, comp, rnd, move=move)
        same = np.all(np.isclose(yd, yh, rtol=1e-12, atol=0), axis=1)
        # a decision within float rounding of its threshold may differ: at most one walker of these few
        assert np.count_nonzero(~same) <= 1
        assert np.allclose(lsd[same], lsh[same], rtol=1e-6, atol=1e-6)
