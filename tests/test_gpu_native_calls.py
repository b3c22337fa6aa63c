"""The operators' calls without ctypes (mimir_b200/csrc/py_ops.cpp) against the general path: the same results, bit for bit, and the same
refusals, for every form of argument that either takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF16, F32 = torch.bfloat16, torch.float32


@pytest.fixture(scope="module")
def T():
    from mimir_b200 import tensor
    return tensor


class _General:
    """Stands in for the module: declines every call."""

    def __getattr__(self, name):
        return lambda *a: None


def forms(shape, dtype):
    """Tensors of one shape in the forms a program may hold them."""
    g = torch.Generator(device="cuda").manual_seed(sum(shape) + len(shape))
    x = torch.randn(shape, generator=g, device="cuda").to(dtype)
    yield "plain", x
    yield "transposed", x.transpose(-1, -2).contiguous().transpose(-1, -2)
    yield "sliced", torch.cat([x, x], -1)[..., :shape[-1]]
    yield "expanded", x[:1].expand(shape)
    yield "offset", torch.cat([x.flatten()[:1], x.flatten()])[1:].view(shape)
    yield "parameter", torch.nn.Parameter(x)
    yield "requires_grad", x.clone().requires_grad_()


def outcome(f):
    try:
        r = f()
        torch.cuda.synchronize()
        return r
    except Exception as e:   # noqa: BLE001 -- the kind of refusal is what is compared
        return type(e)


def same(T, monkeypatch, f):
    got = outcome(f)
    with monkeypatch.context() as m:
        m.setattr(T, "_native", _General())
        want = outcome(f)
    if isinstance(want, type):
        assert got is want
    else:
        assert got.dtype == want.dtype and got.shape == want.shape and got.is_contiguous() == want.is_contiguous()
        assert got.requires_grad == want.requires_grad and torch.equal(got.nan_to_num(7), want.nan_to_num(7))


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("shape", [(1, 1), (3, 5), (24, 16), (2, 3, 4), (3, 40, 24)])
def test_one_operand(T, monkeypatch, dtype, shape):
    gamma = torch.rand(shape[-1], device="cuda") + 0.5
    for name, x in forms(shape, dtype):
        for ax in (0, 1, -1, len(shape), -len(shape) - 1):
            same(T, monkeypatch, lambda: T.reduce("sum", ax, x))
            same(T, monkeypatch, lambda: T.reduce_fused("max", ax, x, "square", outer="abs"))
            same(T, monkeypatch, lambda: T.softmax(ax, x, out_dtype=BF16))
            same(T, monkeypatch, lambda: T.binary_ax("mul", ax, x, x.select(ax, 0) if -len(shape) <= ax < len(shape) else x, then="relu"))
        same(T, monkeypatch, lambda: T.rmsnorm(x, gamma, 1e-6, out_dtype=BF16))
        same(T, monkeypatch, lambda: T.rmsnorm(x, gamma.to(BF16), 1))
        same(T, monkeypatch, lambda: T.unary("tanh", x, out_dtype=F32))
        same(T, monkeypatch, lambda: T.unary("none such", x))
        same(T, monkeypatch, lambda: T.binary("sub", x, x.flip(0)))
        same(T, monkeypatch, lambda: T.binary("sub", x, x[:1]))
        for perm in ((1, 0), (0, 1), (2, 0, 1), [1, 0, 2], (0, 0), (-1, 0)):
            same(T, monkeypatch, lambda: T.transpose(x, perm))
        same(T, monkeypatch, lambda: T.unary("relu", x.cpu()))
        same(T, monkeypatch, lambda: T.unary("relu", x.double()))
        same(T, monkeypatch, lambda: T.softmax(0, x[:0]))


@pytest.mark.parametrize("dtype", [F32, BF16])
@pytest.mark.parametrize("lead,m,n,k", [((), 5, 7, 3), ((), 1, 8, 1), ((), 40, 24, 16), ((3,), 5, 8, 8), ((1,), 4, 1, 2)])
def test_products(T, monkeypatch, dtype, lead, m, n, k):
    run = (lambda *a, **kw: T.bmm(*a, **{q: v for q, v in kw.items() if q == "out_dtype"})) if lead else T.product_2d
    bias = torch.randn(n, device="cuda")
    for _, a in forms(lead + (m, k), dtype):
        for _, b in forms(lead + (k, n), dtype):
            same(T, monkeypatch, lambda: run(a, b))
            same(T, monkeypatch, lambda: run(a, b, post="bias_relu", bias=bias, out_dtype=F32))
        same(T, monkeypatch, lambda: run(a, b, post="bias", bias=bias[:-1]))
        same(T, monkeypatch, lambda: run(a, b, post="bias", bias=bias.to(BF16)))
        same(T, monkeypatch, lambda: run(a, b, post="bias"))
        same(T, monkeypatch, lambda: run(a, b, post="none such"))
        same(T, monkeypatch, lambda: run(a, b.to(F32 if dtype == BF16 else BF16)))
        same(T, monkeypatch, lambda: run(a, b.cpu()))
        same(T, monkeypatch, lambda: run(a[..., :0], b[..., :0, :]))
        same(T, monkeypatch, lambda: run(a, a))


@pytest.mark.parametrize("dtype", [F32, BF16])
def test_attention_and_gated_mlp(T, monkeypatch, dtype):
    for (_, q), (_, k) in zip(forms((2, 3, 17, 64), dtype), forms((2, 3, 30, 64), dtype)):
        for scale, causal in ((0.125, True), (1, False), (1.0, 0)):
            same(T, monkeypatch, lambda: T.attention(q, k, k, scale=scale, causal=causal))
        same(T, monkeypatch, lambda: T.attention(q, q, k))
        same(T, monkeypatch, lambda: T.attention(q[0], k, k))
    for (_, x), (_, w) in zip(forms((9, 64), dtype), forms((64, 64), dtype)):
        same(T, monkeypatch, lambda: T.mlp_gated(x, w, w, w))
        same(T, monkeypatch, lambda: T.mlp_gated(x, w.t(), w.t(), w.t()))
        same(T, monkeypatch, lambda: T.mlp_gated(x, w, w, w.t()))


def test_watched_calls_are_declined(T):
    # a mode or a transform sees the allocation that the general path makes, as it always did
    from torch.utils._python_dispatch import TorchDispatchMode
    x = torch.randn(4, 4, device="cuda")
    assert T._native.unary(T._UNOP["relu"], x, None) is not None
    seen = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))
    with Mode():
        assert T._native.unary(T._UNOP["relu"], x, None) is None
        T.unary("relu", x)
    assert seen
    answers = []
    torch.func.vmap(lambda t: (answers.append(T._native.unary(T._UNOP["relu"], t, None)), t)[1])(x)
    assert answers == [None]


@pytest.mark.parametrize("mode", [torch.enable_grad, torch.no_grad, torch.inference_mode])
def test_the_usual_forms_of_weights_and_modes_are_taken(T, monkeypatch, mode):
    # a program's parameters, and generation in inference mode: taken, with results of the kind that the general path gives
    class Sub(torch.Tensor):
        pass
    x, w = torch.randn((8, 16), device="cuda"), torch.nn.Parameter(torch.randn((16, 24), device="cuda"))
    gamma = torch.nn.Parameter(torch.ones(16, device="cuda"))
    with mode():
        fresh = torch.randn((8, 16), device="cuda")
        for call in (lambda: T._native.product_2d(x, w, T.L.POST_ID, None, None), lambda: T._native.rmsnorm(fresh, gamma, 1e-6, BF16),
                     lambda: T._native.attention(x, x, fresh, 0.25, False), lambda: T._native.unary(T._UNOP["relu"], w, None),
                     lambda: T._native.reduce(T.L.SUM, 0, fresh), lambda: T._native.transpose(w, (1, 0))):
            got = call()
            assert got is not None and type(got) is torch.Tensor and not got.requires_grad
            assert got.is_inference() == torch.is_inference_mode_enabled()
        same(T, monkeypatch, lambda: T.product_2d(fresh, w))
        assert T.product_2d(fresh, w).is_inference() == T.product_2d(fresh, w, full=torch.zeros((8, 24), device="cuda")).is_inference()   # (the general path)
        assert T._native.unary(T._UNOP["relu"], x.as_subclass(Sub), None) is None


def test_other_threads_run_while_a_call_waits(T):
    # the library's buffer grows, which waits for the device: the interpreter's lock is not held meanwhile
    import threading
    import time
    a = torch.randn((8192, 8192), device="cuda").to(BF16)
    small, large = torch.randn((2, 400, 64), device="cuda"), torch.randn((64, 1000, 64), device="cuda")
    ticks, done = [], threading.Event()

    def tick():
        while not done.is_set():
            ticks.append(time.perf_counter())
            time.sleep(1e-3)
    with torch.cuda.stream(torch.cuda.Stream()):
        assert T._native.attention(small, small, small, 0.125, False) is not None
        thread = threading.Thread(target=tick)
        thread.start()
        for _ in range(200):
            T.product_2d(a, a)
        start = time.perf_counter()
        assert T._native.attention(large, large, large, 0.125, False) is not None
        end = time.perf_counter()
        done.set()
        thread.join()
    torch.cuda.synchronize()
    assert end - start > 0.05   # (200 products of 0.8 ms were queued)
    during = [start] + [t for t in ticks if start < t < end] + [end]
    assert max(v - u for u, v in zip(during, during[1:])) < (end - start) / 2
