"""GPU: the calls that go through the native host module give what the general path of ops.py gives, in every form of their arguments, and refuse the
same.  The same kernels run on the same inputs: results are equal bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _Asked:
    """The native module, with a note of whether it served each call (a refusal of the library's is an answer too) or left it to the general path."""

    def __init__(self, host):
        self.host, self.served = host, []

    def __getattr__(self, name):
        def call(*args):
            y = getattr(self.host, name)(*args)
            self.served.append(y is not None)
            return y
        return call


def _same(monkeypatch, f, served=True, raises=None):
    """f() with the native module and without: the same result, or the same error where one is named.  served: whether the module serves the call;
    None: it is not asked."""
    from zhilight_b200 import _lib
    asked, outs = _Asked(_lib.host), []
    for host in (asked, None):
        with monkeypatch.context() as m:
            m.setattr(_lib, "host", host)
            if raises is None:
                outs.append(f())
            else:
                with pytest.raises(raises) as e:
                    f()
                outs.append((type(e.value), getattr(e.value, "code", None)))
    assert asked.served == ([] if served is None else [served])
    a, b = outs
    if raises is not None:
        assert a == b
    else:
        assert a.dtype == b.dtype and a.shape == b.shape and a.stride() == b.stride() and torch.equal(a, b)


class _Own(torch.Tensor):
    pass


# a form of x, whether the native module serves it (None: layers.Linear has refused it before)
FORMS = {"plain": (lambda t: t, True), "strided": (lambda t: torch.cat([t, t], 1)[:, :t.shape[1]], True),
         "parameter": (lambda t: torch.nn.Parameter(t, requires_grad=False), True), "subclass": (lambda t: t.as_subclass(_Own), False),
         "flat": (lambda t: t[0], None), "float": (lambda t: t.float(), None), "narrow": (lambda t: t[:, :64], None)}


def _linear(k, n, quant, dtype, seed):
    from zhilight_b200 import layers
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = torch.randn(n, k, generator=g, device="cuda")
    sd = {"bias": torch.randn(n, generator=g, device="cuda")}
    if quant == 1:
        sd.update(weight=torch.randint(-127, 128, (n, k), generator=g, device="cuda", dtype=torch.int8), weight_scale=torch.rand(n, generator=g, device="cuda") * 0.01)
    elif quant == 7:
        sd.update(weight=w.clamp(-4, 4).to(torch.float8_e4m3fn).view(torch.uint8), weight_scale=torch.tensor([0.1], device="cuda"))
    elif quant == 5:
        sd.update(qweight=torch.randint(-2 ** 31, 2 ** 31 - 1, (k // 8, n), generator=g, device="cuda", dtype=torch.int64).int(),
                  qzeros=torch.full((k // 128, n // 8), 0x77777777, dtype=torch.int32, device="cuda"), scales=torch.rand(k // 128, n, generator=g, device="cuda").half() * 0.01)
    else:
        sd["weight"] = w * 0.05
    lin = layers.Linear(k, n, "", quant, dtype)
    lin.load_state_dict(sd)
    return lin, g


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("m", [1, 40])
def test_linears(lib, cuda, monkeypatch, form, m):
    from zhilight_b200 import ZLError
    make, served = FORMS[form]
    for quant, dtype in ((0, "bfloat"), (0, "half"), (1, "half"), (7, "bfloat"), (5, "half")):
        lin, g = _linear(512, 384, quant, dtype, m)
        x = torch.randn(m, 512, generator=g, device=cuda).to(lin.dtype)
        _same(monkeypatch, lambda: lin(make(x)), served, ZLError if served is None else None)
        _same(monkeypatch, lambda: lin(x[None]))


ONE_ROW = {"odd pitch": lambda x: torch.cat([x, x[:, :13]], 1).expand(2, -1).contiguous()[:1, :x.shape[1]], "pitch of one": lambda x: x.flatten().as_strided(x.shape, (1, 1)),
           "short pitch": lambda x: x.flatten().as_strided(x.shape, (8, 1)), "broadcast": lambda x: x.expand(1, -1).as_strided(x.shape, (0, 1))}


@pytest.mark.parametrize("form", sorted(ONE_ROW))
@pytest.mark.parametrize("quant,dtype", [(0, "bfloat"), (0, "half"), (1, "half"), (7, "bfloat"), (5, "half")])
def test_one_row_of_any_pitch(lib, cuda, form, quant, dtype):
    """A single row is contiguous whatever lies between it and a next one that is not there."""
    lin, g = _linear(512, 384, quant, dtype, 3)
    x = torch.randn(1, 512, generator=g, device=cuda).to(lin.dtype)
    given = ONE_ROW[form](x)
    assert given.stride(0) != 512 and torch.equal(given, x)
    assert torch.equal(lin(given), lin(x))


def test_entry_points(lib, cuda, monkeypatch):
    from zhilight_b200 import ZLError, ops
    g = torch.Generator(device="cuda").manual_seed(0)
    x, w = torch.randn(3, 256, generator=g, device=cuda).half(), torch.randn(512, 256, generator=g, device=cuda).half()
    scale = torch.rand(512, device=cuda, generator=g)
    packed = torch.zeros(int(lib.zl_w4_packed_bytes(512, 256, 128)), dtype=torch.uint8, device=cuda)
    given = torch.empty(3, 512, device=cuda).half()
    _same(monkeypatch, lambda: ops.w4a16_gemm_fused(x, packed, 512, 256, variant=1))
    _same(monkeypatch, lambda: ops.w4a16_gemm_fused(x, packed, 512, 256, variant=1, out=given))
    _same(monkeypatch, lambda: ops.w4a16_gemm_fused(x, packed, 512, 256, epilogue=ops.EPI_SWIGLU, variant=1, pdl=True))
    _same(monkeypatch, lambda: ops.w4a16_gemm_fused(x, packed, 512, 256, epilogue=ops.EPI_RESIDUAL, variant=1), raises=ZLError)
    _same(monkeypatch, lambda: ops.w4a16_gemm_fused(x.float(), packed, 512, 256, variant=1), False, ZLError)
    _same(monkeypatch, lambda: ops.dense_gemm_skinny(x, w, out_dtype=torch.float32))
    _same(monkeypatch, lambda: ops.dense_gemm_skinny(x, w, out_dtype=torch.float64), False, ZLError)
    _same(monkeypatch, lambda: ops.dense_gemm_skinny(x, w.t()), False, ZLError)
    _same(monkeypatch, lambda: ops.dense_gemm_skinny(x[:, :7].contiguous(), w[:, :7].contiguous()), raises=ZLError)
    _same(monkeypatch, lambda: ops.dense_gemm_skinny(x.cpu(), w), False, ZLError)
    _same(monkeypatch, lambda: ops.int8_linear(x, w.to(torch.int8), scale))
    _same(monkeypatch, lambda: ops.int8_linear(x[:0], w.to(torch.int8), scale), raises=ZLError)
    _same(monkeypatch, lambda: ops.fp8_linear(x, w.to(torch.float8_e4m3fn).view(torch.uint8), torch.ones(1, device=cuda)))
    _same(monkeypatch, lambda: ops.fp8_linear(x, w.to(torch.int8), torch.ones(1, device=cuda).double()), False, ZLError)


@pytest.mark.parametrize("b,len_q", [(1, 1), (5, 1), (1, 40)])
def test_attention(lib, cuda, monkeypatch, b, len_q):
    from zhilight_b200 import ZLError, ops
    g = torch.Generator(device="cuda").manual_seed(b)
    lens = [300 - 17 * i for i in range(b)]
    q = torch.randn(b, len_q, 8, 128, generator=g, device=cuda).half()
    ks, vs = ([torch.randn(n, 2, 128, generator=g, device=cuda).half() for n in lens] for _ in range(2))
    length = torch.tensor(lens, dtype=torch.int32, device=cuda)
    mask = torch.ones(len_q, lens[0], device=cuda).tril(lens[0] - len_q).to(torch.int8) if len_q > 1 else None

    def call(k=ks, v=vs, m=mask, scale=0.09, query=q, pdl=False):
        return ops.decode_attention(query, length, k, v, m, scale, max(lens), 2, pdl=pdl)
    for f in (call, lambda: call(tuple(ks), tuple(vs)), lambda: call(scale=1), lambda: call(pdl=True)):
        _same(monkeypatch, f)
    for f in (lambda: call([t.as_subclass(_Own) for t in ks]), lambda: call([torch.from_dlpack(t) for t in ks])):
        _same(monkeypatch, f, False)
    _same(monkeypatch, lambda: call(iter(ks), list(vs)), False, TypeError)
    _same(monkeypatch, lambda: call(query=torch.cat([q, q], 3)[..., :128]), False, ZLError)
    _same(monkeypatch, lambda: call(query=q.double()), False, ZLError)
    _same(monkeypatch, lambda: call(query=q[0]), False, ValueError)


def test_memory_of_another_stream_outlives_its_tensors(lib, cuda):
    """A cache that was allocated on another stream and dropped at once is not given away before the call has read it."""
    from zhilight_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(0)
    n = 4096
    q = torch.randn(1, 1, 8, 128, generator=g, device=cuda).half()
    k, v = (torch.randn(n, 2, 128, generator=g, device=cuda).half() for _ in range(2))
    length = torch.tensor([n], dtype=torch.int32, device=cuda)
    ref = ops.decode_attention(q, length, [k], [v], None, 0.09, n, 2)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        k2, v2 = k.clone(), v.clone()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda._sleep(20_000_000)
    out = ops.decode_attention(q, length, [k2], [v2], None, 0.09, n, 2)
    at = {k2.data_ptr(), v2.data_ptr()}
    del k2, v2
    with torch.cuda.stream(side):
        new = [torch.full_like(k, 7.0) for _ in range(4)]
    assert not at & {t.data_ptr() for t in new}
    torch.cuda.synchronize()
    assert torch.equal(out, ref)


@pytest.mark.parametrize("call", ["w4", "dense", "int8", "attention"])
@pytest.mark.parametrize("native", [True, False])
def test_out_of_memory_is_torchs_own_error(lib, cuda, monkeypatch, call, native):
    """A program that frees memory and tries again knows it by its type.  No kernel is launched: the result cannot be allocated."""
    from zhilight_b200 import _lib, ops
    assert _lib.host is not None
    m, n, k = 2048, 32768, 128
    x, w = torch.zeros(m, k, device=cuda).half(), torch.zeros(n, k, device=cuda, dtype=torch.int8)
    packed = torch.zeros(int(lib.zl_w4_packed_bytes(n, k, 128)), dtype=torch.uint8, device=cuda)
    wh, one = torch.zeros(n, k, device=cuda).half(), torch.ones(n, device=cuda)
    q, kv = torch.zeros(1, 4096, 128, 128, device=cuda).half(), torch.zeros(4096, 1, 128, device=cuda).half()
    lens = torch.tensor([4096], dtype=torch.int32, device=cuda)
    run = {"w4": lambda: ops.w4a16_gemm_fused(x, packed, n, k, variant=1), "dense": lambda: ops.dense_gemm_skinny(x, wh),
           "int8": lambda: ops.int8_linear(x, w, one), "attention": lambda: ops.decode_attention(q, lens, [kv], [kv], None, 0.09, 4096, 1)}[call]
    if not native:
        monkeypatch.setattr(_lib, "host", None)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(1e-6)
    try:
        with pytest.raises(torch.OutOfMemoryError):
            run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
