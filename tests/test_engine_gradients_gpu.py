"""The sharded decoder engine's gradients on one GPU, against the plain PyTorch decoder on the CPU (fp32)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda", 0)


def _source(**over):
    """A small decoder whose biases and norm weights are not their initial zeros and ones, every weight a bf16 value."""
    from odc_b200.models import DecoderLM, get_config
    cfg = get_config("tiny", **over)
    src = DecoderLM(cfg)
    src.reset_parameters(seed=0)
    gen = torch.Generator().manual_seed(5)
    with torch.no_grad():
        for name, p in src.named_parameters():
            if "norm" in name:
                p.normal_(1.0, 0.1, generator=gen)
            elif "bqkv" in name:
                p.normal_(0.0, 0.05, generator=gen)
            p.copy_(p.bfloat16())
    return cfg, src


def _batches(cfg, n=2, lo=16, hi=128, tokens=512, seed=0):
    from odc_b200.data import LengthSpec, make_minibatch
    return make_minibatch(0, 0, cfg.vocab_size, LengthSpec("uniform", lo=lo, hi=hi), n, tokens, seed=seed)


def _args(mb):
    return mb["input_ids"], mb["position_ids"], mb["cu_seqlens"], mb["max_seqlen"]


class _Engine:
    def __init__(self, **over):
        import odc_b200 as odc
        from odc_b200.parallel import FusedDecoderLM
        self.cfg, self.src = _source(**over)
        odc.init_nvshmem(DEV, 2 << 30)
        self.model = FusedDecoderLM(self.cfg, device=DEV, source=self.src)

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.model.stop()

    def minibatch(self, mbs, factor=1.0, sync=None):
        """One minibatch; the accumulators by parameter name.  ``sync``: synchronisation on or off per microbatch."""
        from odc_b200.data import to_device
        self.model.start_minibatch()
        for i, mb in enumerate(mbs):
            if sync is not None:
                self.model.set_requires_gradient_sync(sync[i])
            mb = to_device(mb, DEV)
            (factor * self.model(*_args(mb), labels=mb["labels"], loss_scale=mb["loss_scale"])).backward()
        self.model.finish_minibatch()
        return self.grads()

    def grads(self):
        out = {name: p.grad()[:p.out_features].clone() for name, p in self.model.matrices().items()}
        out.update({name: self.model.small.acc[o:o + n].clone() for name, (o, n) in self.model.small.slots.items()})
        return out


# About 20 values on the way through a layer and back are rounded to bf16 (2^-9 each, P and dS of the attention among them);
# with two layers and the head some 50 independent roundings, sqrt(50) * 2^-9 = 1.4e-2 of a gradient's norm at most.
CHAIN = 2e-2


def _rel(got, want):
    want = want.double()
    return ((got.double().to(want.device).reshape(want.shape) - want).norm() / want.norm()).item()


def test_gradients_of_an_abandoned_pass_do_not_reach_the_next_minibatch():
    """A backward that raised half way has already added the norm gradients of the layers behind it."""
    from odc_b200.data import to_device
    with _Engine() as e:
        mbs = _batches(e.cfg)
        clean = e.minibatch(mbs)
        mb = to_device(mbs[0], DEV)

        def fail(grad):
            raise RuntimeError("abandoned")

        handle = e.model.layers[0].register_forward_hook(lambda mod, args, out: out.register_hook(fail) and None)
        e.model.start_minibatch()
        with pytest.raises(RuntimeError, match="abandoned"):
            e.model(*_args(mb), labels=mb["labels"], loss_scale=mb["loss_scale"]).backward()
        handle.remove()
        again = e.minibatch(mbs)
        for name, want in clean.items():   # the same sums, in another order of additions
            assert _rel(again[name], want) < 1e-3, name


@pytest.mark.parametrize("route", ["tma", "red", "other nodes"])
def test_qkv_bias_gradient_on_every_route(monkeypatch, route):
    """The native layer adds the bias gradient in its kernel; the Python layer runs with per-thread reductions asked for,
    and in groups whose rows are not all mapped here."""
    from odc_b200.parallel import ShardedParameter
    if route == "other nodes":
        monkeypatch.setattr(ShardedParameter, "reaches_other_nodes", lambda self: True)
    else:
        monkeypatch.setenv("ODC_WGRAD_SCATTER", route)
    with _Engine(qkv_bias=True, tie_embeddings=True) as e:
        mbs = _batches(e.cfg)
        got = e.minibatch(mbs)
        for mb in mbs:
            e.src(*_args(mb), labels=mb["labels"], loss_scale=mb["loss_scale"]).backward()
        for name, p in e.src.named_parameters():
            assert _rel(got[name], p.grad) < CHAIN, name


@pytest.mark.parametrize("leaf", [False, True])
def test_a_layer_on_its_own(leaf):
    """A layer that is called with activations of its own, which need a gradient or not, still gets all its gradients."""
    with _Engine(qkv_bias=True) as e:
        mb = _batches(e.cfg, n=1)[0]
        where = tuple(t.to(DEV) if torch.is_tensor(t) else t for t in _args(mb)[1:])
        T = mb["input_ids"].numel()
        gen = torch.Generator().manual_seed(9)
        x = torch.randn(T, e.cfg.hidden_size, generator=gen).bfloat16()
        dy = torch.randn(T, e.cfg.hidden_size, generator=gen).bfloat16()
        e.model.start_minibatch()
        e.model.layers[0](x.to(DEV).requires_grad_(leaf), *where).backward(dy.to(DEV))
        e.model.finish_minibatch()
        got = e.grads()
        e.src.layers[0](x.float(), *_args(mb)[1:]).backward(dy.float())
        for name, p in e.src.layers[0].named_parameters():
            assert _rel(got[f"layers.0.{name}"], p.grad) < CHAIN, name


@pytest.mark.parametrize("switch", ["ODC_DETERMINISTIC", "torch"])
def test_embedding_gradient_is_reproducible_where_that_is_asked_for(monkeypatch, switch):
    """A tied matrix gets the head's gradient and rows of the lookup, many for one token: with either switch they are
    added in one order.  Sequences of one key tile: the attention's own sums over key tiles have no fixed order."""
    if switch == "ODC_DETERMINISTIC":   # per-producer slots, and column sums in a fixed order
        monkeypatch.setenv(switch, "1")
    torch.use_deterministic_algorithms(True)
    try:
        with _Engine(tie_embeddings=True) as e:
            mbs = _batches(e.cfg, lo=64, hi=128, tokens=2048)
            for mb in mbs:
                mb["input_ids"] = mb["input_ids"] % 3
            runs = [e.minibatch(mbs)["embed.weight"] for _ in range(6)]
            same = [torch.equal(runs[0], r) for r in runs[1:]]
    finally:
        torch.use_deterministic_algorithms(False)
    assert all(same), same


@pytest.mark.parametrize("form", ["int32", "strided"])
def test_token_ids_of_any_integer_form(form):
    """Ids as 32-bit integers or as a column of a wider array: the gradients of plain contiguous ids."""
    from odc_b200.data import to_device
    with _Engine(tie_embeddings=True) as e:
        mb = to_device(_batches(e.cfg, n=1)[0], DEV)
        ids = mb["input_ids"]
        other = {"int32": ids.int(), "strided": torch.stack([ids, ids + 1], 1)[:, 0]}[form]

        def grads(ids):
            e.model.start_minibatch()
            x = e.model.hidden_states(ids, *_args(mb)[1:])
            x.backward(torch.ones_like(x))
            e.model.finish_minibatch()
            return e.grads()["embed.weight"]

        want, got = grads(ids), grads(other)
        assert want.norm() > 0 and _rel(got, want) < 1e-3


def test_passes_on_another_stream_than_the_start_of_their_minibatch():
    """They find cleared accumulators and the weights of an optimizer step that was still running when it returned."""
    from odc_b200.data import to_device
    with _Engine(qkv_bias=True) as e:
        mbs = _batches(e.cfg)
        clean = e.minibatch(mbs)
        on_device = [to_device(mb, DEV) for mb in mbs]
        other = torch.cuda.Stream()
        groups = e.model.optimizer_groups()
        for g in groups:
            g.flat()[4].zero_()
        torch.cuda.synchronize()
        torch.cuda._sleep(50_000_000)        # some 25 ms
        for g in groups:                     # the optimizer's writes
            g.flat()[4].copy_(g.flat()[0])
        e.model.start_minibatch()
        with torch.cuda.stream(other):
            for mb in on_device:
                e.model(*_args(mb), labels=mb["labels"], loss_scale=mb["loss_scale"]).backward()
        torch.cuda.current_stream().wait_stream(other)
        e.model.finish_minibatch()
        got = e.grads()
        for name, want in clean.items():     # the same sums, in another order of additions
            assert _rel(got[name], want) < 1e-3, name


@pytest.mark.parametrize("tied", [True, False])
def test_activation_gradients_do_not_depend_on_deferral(tied):
    """A loss factor that bf16 cannot hold (1/3, off by 2^-9 when rounded): the layers' gradients of a microbatch are the
    same whether its weight gradients are pushed at once or held back.  Both forms round the same bf16 activations, so the
    difference is that of fp32 sums."""
    with _Engine(tie_embeddings=tied) as e:
        mbs = _batches(e.cfg, n=2, lo=64, hi=128)   # one key tile per sequence: no sums in a free order
        now = e.minibatch(mbs, factor=1 / 3)
        held = e.minibatch(mbs, factor=1 / 3, sync=[False, True])
        for name, want in now.items():
            assert _rel(held[name], want) < 1e-4, name


@pytest.mark.parametrize("sync", [None, [False, True], [True, False]])
@pytest.mark.parametrize("tied,bias", [(True, True), (False, False)])
def test_every_accumulator_matches_the_plain_decoder(tied, bias, sync):
    """Two microbatches with a loss factor, pushed at once, or held back and handed to the Python layer, tied and untied
    heads: every accumulator after the minibatch is the gradient of the plain decoder."""
    with _Engine(qkv_bias=bias, tie_embeddings=tied) as e:
        mbs = _batches(e.cfg)
        got = e.minibatch(mbs, factor=0.75, sync=sync)
        for mb in mbs:
            (0.75 * e.src(*_args(mb), labels=mb["labels"], loss_scale=mb["loss_scale"])).backward()
        want = dict(e.src.named_parameters())
        assert set(got) == set(want)
        for name, p in want.items():
            assert _rel(got[name], p.grad) < CHAIN, name


@pytest.mark.parametrize("subclass", [False, True])
@pytest.mark.parametrize("chunk,kept", [(4096, True), (300, False)])
def test_hidden_states_may_be_written_to_after_the_loss(chunk, kept, subclass):
    """One chunk, whose products wait for the backward, and several: what the loss needs of the hidden states is its own."""
    from odc_b200 import ops
    with _Engine() as e:
        e.cfg.ce_chunk = e.model.cfg.ce_chunk = chunk
        mbs = _batches(e.cfg, n=1, lo=64, hi=128)   # one key tile per sequence: no sums in a free order
        states, calls = [], []
        plain, loss = e.model.hidden_states, ops._ext().loss_and_logit_grads
        holds = lambda *a: states.append(plain(*a)) or states[-1]
        if subclass:
            e.model.__class__ = type("Holds", (type(e.model),), {"hidden_states": lambda self, *a: holds(*a)})
        else:
            e.model.hidden_states = holds
        want = e.minibatch(mbs)
        whole = type(e.model).forward

        def forward(*args, **kw):
            out = whole(e.model, *args, **kw)
            states[-1].data.zero_()
            with torch.no_grad():
                states[-1].add_(1)
            return out
        e.model.forward = forward
        ops._ext().loss_and_logit_grads = lambda *a: calls.append(1) or loss(*a)
        try:
            got = e.minibatch(mbs)
        finally:
            ops._ext().loss_and_logit_grads = loss
        assert len(states) == 2 and bool(calls) == kept
        for name in want:   # the same sums, in another order of additions
            assert _rel(got[name], want[name]) < 1e-3, name


@pytest.mark.parametrize("library", [False, True])
@pytest.mark.parametrize("add", [False, True])
def test_head_gradients_for_a_buffer_that_is_pushed_later(monkeypatch, add, library):
    """What several ranks push, the matrix without the loss gradient, and what is held back, the sum with it; together in one launch,
    and one by one with library products.  Against 64 bits."""
    from odc_b200 import ops
    with _Engine() as e:
        p = e.model.head_param()
        w = e.model.head_full()[:p.out_features]
        torch.manual_seed(0)
        T, V, H = 300, w.shape[0], w.shape[1]
        d, h = (0.01 * torch.randn(T, V, device=DEV)).bfloat16(), torch.randn(T, H, device=DEV).bfloat16()
        g = torch.tensor(1 / 3, device=DEV)
        local = torch.randn(V, H, device=DEV)
        start = local.double()
        matrix = p.matrix()
        if library:
            monkeypatch.setenv("ODC_GEMM", "cublas")
        dh = ops._ext().sharded_head_grads(d, h, w, g, matrix, local, add)
        want_dh, want = d.double() @ w.double() / 3, d.double().t() @ h.double()
        term = want / 3 if add else want
        want = start + term if add else term
        # one rounding to bf16 (one by one, two), fp32 sums of 300 to 1024 products; a library product is rounded to bf16 whatever it is for
        assert ((dh.double() - want_dh).abs() <= 2 ** -7 * want_dh.abs() + 1e-5).all()
        rounded = 2 ** -8 if library else 2 ** -20
        assert ((local.double() - want).abs() <= rounded * term.abs() + 2 ** -20 * start.abs() + 1e-5).all()


class _Counting(torch.nn.Module):
    def __init__(self, inner, calls):
        super().__init__()
        self.inner, self.calls, self.weight = inner, calls, inner.weight   # what the engine asks its layers for

    def forward(self, *args, **kw):
        self.calls.append(1)
        return self.inner(*args, **kw)


@pytest.mark.parametrize("form", ["hook", "global hook", "replaced"])
@pytest.mark.parametrize("name", ["w_gate_up", "w_down"])
def test_layers_of_the_mlp_are_called_where_somebody_stands_between(form, name):
    """The MLP takes its two matrices as one function, but not past a module hook or a module put in a layer's place."""
    with _Engine() as e:
        mbs = _batches(e.cfg, lo=64, hi=128)   # one key tile per sequence: no sums in a free order
        clean = e.minibatch(mbs)
        layer, calls, handle = e.model.layers[1], [], None
        inner = getattr(layer, name)
        if form == "hook":
            inner.register_forward_hook(lambda *args: calls.append(1))
        elif form == "global hook":
            handle = torch.nn.modules.module.register_module_forward_hook(lambda m, *args: calls.append(1) if m is inner else None)
        else:
            setattr(layer, name, _Counting(inner, calls))
        try:
            got = e.minibatch(mbs)
        finally:
            if handle is not None:
                handle.remove()
        assert len(calls) == len(mbs)
        for key, want in clean.items():   # the same roundings; fp32 sums of products in another order
            assert _rel(got[key], want) < 1e-3, key


@pytest.mark.parametrize("name,tokens", [("llama3.2-1b", [5, 128, 77]), ("qwen2.5-1.5b", [300, 64]), ("tiny", [1])])
@pytest.mark.parametrize("grad", [True, False])
def test_a_layer_as_one_function_is_its_parts(name, tokens, grad):
    """The same roundings: the same bytes forward; backward the additions of the norms' and the queries' gradients come in any
    order (fp32, then rounded to bf16: 2^-8 of what a flipped rounding moves, far less in the norm)."""
    from odc_b200 import ops
    from odc_b200.models import DecoderLayer, get_config
    cfg = get_config(name)
    cfg.num_layers = 1
    torch.manual_seed(0)
    with torch.device("cuda"):
        layer = DecoderLayer(cfg).bfloat16()
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0 if p.dim() == 2 else 0.5, 0.05)
    T = sum(tokens)
    x = torch.randn(T, cfg.hidden_size, device="cuda").bfloat16().requires_grad_(grad)
    for p in layer.parameters():
        p.requires_grad_(grad)
    dy = torch.randn(T, cfg.hidden_size, device="cuda").bfloat16()
    pos = torch.cat([torch.arange(n) for n in tokens]).cuda()
    cu = torch.tensor([0] + tokens).cumsum(0).int().cuda()
    taken = []
    whole = ops.decoder_layer
    results = []
    for parts in (False, True):
        ops.decoder_layer = (lambda *a: None) if parts else (lambda *a: taken.append(whole(*a)) or taken[-1])
        try:
            y = layer(x, pos, cu, max(tokens))
        finally:
            ops.decoder_layer = whole
        results.append([y] + (list(torch.autograd.grad(y, [x, *layer.parameters()], dy)) if grad else []))
    assert len(taken) == 1 and taken[0] is not None
    assert torch.equal(results[0][0], results[1][0])
    for a, b in zip(*results):
        assert a.dtype == b.dtype and a.shape == b.shape and _rel(a.float(), b.float()) < 3e-3


def test_layers_that_are_not_taken_as_one_function():
    """A frozen weight, weights of other types, strided activations and three dimensions go through the parts as before."""
    from odc_b200 import ops
    from odc_b200.models import DecoderLayer, get_config
    cfg = get_config("llama3.2-1b")
    with torch.device("cuda"):
        layer = DecoderLayer(cfg).bfloat16()
    with torch.no_grad():
        for p in layer.parameters():
            p.normal_(0.0, 0.02)
    x = torch.randn(300, cfg.hidden_size, device="cuda").bfloat16()
    pos, cu = torch.arange(300, device="cuda"), torch.tensor([0, 300], dtype=torch.int32, device="cuda")
    want = layer(x, pos, cu, 300)
    layer.mlp.w_down.requires_grad_(False)
    y = layer(x.requires_grad_(), pos, cu, 300)
    assert torch.equal(y, want)
    y.sum().backward()
    assert layer.mlp.w_down.grad is None and layer.mlp.w_gate_up.grad is not None and x.grad is not None
    layer.mlp.w_down.requires_grad_(True)
    with torch.no_grad():
        strided = torch.empty(300, 2 * cfg.hidden_size, device="cuda", dtype=torch.bfloat16)[:, :cfg.hidden_size]
        strided.copy_(x)
        assert torch.equal(layer(strided, pos, cu, 300), want)
