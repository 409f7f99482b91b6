"""The tcgen05 form of the weight-streaming product: tile edges, remainders of K and tokens, every epilogue."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(m, n, k, dual, split, seed=0, pad=0):
    g = torch.Generator().manual_seed(seed)
    ri = lambda *s: torch.randint(-128, 128, s, generator=g, dtype=torch.int8)
    # rows of the activations lie in a wider tensor, like the latents of a pair
    wide = ri(m, (2 if split else 1) * k + 16 * pad).cuda()
    d = dict(a=wide[:, :k], w=ri(n, k).cuda(), sa=(torch.rand(m, generator=g) * 1e-2 + 1e-3).cuda(),
             ws=(torch.rand(n, generator=g) * 1e-2 + 1e-3).cuda())
    if dual:
        d.update(w2=ri(n, k).cuda(), ws2=(torch.rand(n, generator=g) * 1e-2 + 1e-3).cuda())
    if split:
        d.update(a2=wide[:, k:2 * k], sa2=(torch.rand(m, generator=g) * 1e-2 + 1e-3).cuda())
    return d


SHAPES = [(1, 16, 16), (3, 48, 80), (4, 128, 128), (5, 144, 256), (16, 1024, 4096), (17, 272, 496), (29, 5504, 512), (32, 64, 2048),
          (33, 208, 1040), (47, 4096, 384), (48, 112, 2064), (63, 4112, 1024), (64, 2560, 528), (64, 32, 16384)]


@pytest.mark.parametrize("m,n,k", SHAPES)
@pytest.mark.parametrize("kind", ["single", "dual", "split"])
def test_accumulators_and_results(m, n, k, kind):
    """int32 sums against float64 (exact: |sum| < 2**53), fp16 results and the all-fp32 epilogue's row maxima bit for bit
    against the register-fed form, which shares nothing with this one but the epilogue's statement."""
    from lsvd_b200.ffn import w8a8_gemv
    dual, split = kind != "single", kind == "split"
    d = _case(m, n, k, dual, split, seed=m + n, pad=1)
    kw = dict(w2_q=d["w2"], w2_scale=d["ws2"]) if dual else {}
    if split:
        kw.update(a2_q=d["a2"], a2_scale=d["sa2"])
    res = torch.randn(m, n + 3, device="cuda").half()[:, 1:n + 1] if not dual else None      # odd stride, 2-byte aligned
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    buf = [torch.zeros(m, n + 5, dtype=torch.float16, device="cuda") for _ in range(2)]
    got = w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], want_acc=True, residual=res, out=buf[0], out_col=3, status_word=status, form=4, **kw)
    want = w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], want_acc=True, residual=res, out=buf[1], out_col=3, form=3, **kw)
    assert int(status) == 0
    exact = d["a"].double() @ d["w"].double().t()
    assert torch.equal(got[1].double(), exact)
    if dual:
        a2 = d["a2"] if split else d["a"]
        assert torch.equal(got[2].double(), a2.double() @ d["w2"].double().t())
    assert torch.equal(buf[0], buf[1])                                     # untouched border columns included
    if not dual:
        o32 = [torch.empty(m, n, device="cuda") for _ in range(2)]
        w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], want_out=False, out_f32=o32[0], form=4)
        w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], want_out=False, out_f32=o32[1], form=3)
        assert torch.equal(o32[0], o32[1])
    words = [torch.zeros(m, 4, dtype=torch.int32, device="cuda") for _ in range(2)]
    outs = [w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], fp32_swiglu=dual, row_absmax=words[i], absmax_split=16 if n > 16 else 0,
                      form=4 - i, prefetch_weights=2 * (i == 0), **kw)[0] for i in range(2)]
    assert torch.equal(outs[0], outs[1])
    assert torch.equal(words[0], words[1])


@pytest.mark.parametrize("m,n,k,dual", [(1, 4096, 512, False), (8, 256, 8192, False), (8, 256, 8176, False), (9, 16384, 256, False), (9, 16368, 256, False),
                                        (17, 16384, 16, False), (17, 8192, 4096, False), (16, 8192, 4096, False), (33, 1024, 4096, False), (33, 1008, 4096, False), (33, 1024, 1024, True),
                                        (33, 1008, 1024, True)])
def test_the_form_chosen_by_size_has_the_same_bits(m, n, k, dual):
    """Both sides of each line of the choice: without a hint, with one, and with the early read (nothing wrote the weights)."""
    from lsvd_b200.ffn import w8a8_gemv
    d = _case(m, n, k, dual, False, seed=n)
    kw = dict(w2_q=d["w2"], w2_scale=d["ws2"]) if dual else {}
    want = w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], want_acc=True, form=3, **kw)
    torch.cuda.synchronize()
    for early in (False, True, 2):
        got = w8a8_gemv(d["a"], d["sa"], d["w"], d["ws"], want_acc=True, prefetch_weights=early, **kw)
        for x, y in zip(got, want):
            assert x is y is None or torch.equal(x, y)


@pytest.mark.parametrize("early", [False, 2])
@pytest.mark.parametrize("m,n,k", [(1, 256, 8192), (5, 64, 512), (29, 64, 8192), (64, 1024, 4096)])
def test_broadcast_and_overlapping_rows(m, n, k, early):
    """Rows that no tensor map describes -- one activation row for all tokens, windows of one buffer as weights, any stride of a
    single row -- give what their contiguous copies give, also where the size alone would choose the tcgen05 kernel."""
    from lsvd_b200.ffn import w8a8_gemv
    d = _case(m, n, k, False, False, seed=k)
    one = d["a"][:1].contiguous().expand(m, k) if m > 1 else d["a"].contiguous().as_strided((1, k), (16, 1))
    windows = torch.randint(-128, 128, (16 * n + k,), dtype=torch.int8, device="cuda").as_strided((n, k), (16, 1))
    for a, w in ((one, d["w"]), (d["a"], windows), (one, windows)):
        got = w8a8_gemv(a, d["sa"], w, d["ws"], want_acc=True, prefetch_weights=early)
        want = w8a8_gemv(a.contiguous(), d["sa"], w.contiguous(), d["ws"], want_acc=True, form=3)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    with pytest.raises(ValueError):
        w8a8_gemv(d["a"], d["sa"], windows, d["ws"], form=4)


@pytest.mark.parametrize("form", [0, 3, 4])
def test_hint_behind_the_kernel_that_writes_the_weights(form):
    """``prefetch_weights=True`` is a hint wherever the call stands, directly behind a copy into the weights too."""
    from lsvd_b200.ffn import w8a8_gemv
    d = _case(8, 4096, 8192, False, False, seed=3)
    other = _case(8, 4096, 8192, False, False, seed=4)["w"]
    want = [w8a8_gemv(d["a"], d["sa"], w.clone(), d["ws"], form=3)[0] for w in (d["w"], other)]
    w = d["w"].clone()
    got = []
    for i in range(20):
        w.copy_(other if i % 2 else d["w"])
        got.append(w8a8_gemv(d["a"], d["sa"], w, d["ws"], form=form, prefetch_weights=True)[0])
    assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))


@pytest.mark.parametrize("graph", [False, True])
def test_weights_rewritten_on_the_stream_right_before_a_step(graph):
    """A step whose products read weights before their wait sees what was written to them in front of its first quantiser: the
    hybrid FFN (both streams) and the mixffn structure, eager and captured with the copies."""
    from lsvd_b200 import synth
    from lsvd_b200.ffn import HybridFFN
    from lsvd_b200.mixffn import MixedFFNGateUpDenseLatentFused
    from oracle import mixffn as omix
    hk = synth.sign_matrix(12, seed=0).float()
    cuda = lambda w: {k: v.cuda() if isinstance(v, torch.Tensor) else v for k, v in w.items()}
    gen = torch.Generator().manual_seed(4)
    mk = lambda o, i: (torch.randn(o, i, generator=gen) / i ** 0.5).half()
    mix = lambda: omix.convert_swiglu(mk(1024, 512), mk(1024, 512), mk(512, 1024), torch.randn(512, generator=gen).half(), 0.5, 0.5, 64, gen)
    for make, ws in ((HybridFFN, [synth.ffn_weights(1024, 12 * 64, 128, 384, seed=s, had_K=hk, K=12) for s in (1, 2)]),
                     (MixedFFNGateUpDenseLatentFused, [mix(), mix()])):
        mods = [make(cuda(w)) for w in ws]
        live = make(cuda(ws[0]))
        x = torch.randn(5, 1024 if make is HybridFFN else 512, generator=gen).half().cuda()
        want = [m(x).clone() for m in mods]
        assert not torch.equal(*want)

        def step(i):
            for mine, given in zip(live.buffers(), mods[i].buffers()):
                mine.copy_(given)
            return live(x)
        if graph:
            step(0)
            torch.cuda.synchronize()
            graphs = []
            for i in range(2):
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    y = step(i)
                graphs.append((g, y))
            for _ in range(10):
                for i, (g, y) in enumerate(graphs):
                    g.replay()
                    assert torch.equal(y, want[i])
        else:
            got = [step(i % 2).clone() for i in range(20)]
            assert all(torch.equal(y, want[i % 2]) for i, y in enumerate(got))
