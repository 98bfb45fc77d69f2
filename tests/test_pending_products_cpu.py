"""Which parts hand a sublayer's last product, or rows without their norm's factors, to one another: the parts of the package among
themselves, and nobody else. Runs on the CPU: with the plain kernel table, which has no such product, and with one that restates
it."""
from functools import wraps

import numpy as np
import pytest
import torch

from fusezap_core_b200.cache import CacheManager
from fusezap_core_b200.config import LayerSpec, ModelSpec, PartSpec, ScheduleEntry
from fusezap_core_b200.engine import Portion, StepRunner
from fusezap_core_b200.engine.model import DecoderModel
from fusezap_core_b200.kernels.interface import ScaledRows
from fusezap_core_b200.parts import BLOCKS, FEED_FORWARDS, MIXERS, NORMS, POSITIONS
from fusezap_core_b200.parts.attention import GQAttention
from fusezap_core_b200.parts.base import PendingProduct
from fusezap_core_b200.parts.block import PreNormBlock
from fusezap_core_b200.parts.feed_forward import SwiGLU
from fusezap_core_b200.parts.norm import RMSNorm
from fusezap_core_b200.parts.rope import RotaryEncoding
from plain_ops import PlainOps

D, V, EPS = 32, 61, 1e-5
IDS = [[int(t) for t in np.random.default_rng(n).integers(0, V, n)] for n in (9, 4)]


class Plain(PlainOps):
    def embed(self, table, tokens, x, src=None, prev_ids=None, scale=1.0, copy=None):
        super().embed(table, tokens, x, src, prev_ids, scale)
        if copy is not None:
            copy.copy_(x)

    def weighted_sum(self, terms, weights, out):
        out.copy_(sum(t * w for t, w in zip(terms, weights)))


class FoldingOps(Plain):
    """The plain table with a product that ends in the residual add and the norm, and products that read its rows."""
    parts = 4

    def __init__(self):
        super().__init__()
        self.folded = self.scaled_products = 0

    def norm_parts(self, m, n, k):
        return self.parts

    def linear_add_norm(self, a, w, bias, x, weight, h, squares):
        x += a.float() @ w.float().T + (0 if bias is None else bias)
        h.copy_((x * weight.float()).to(h.dtype))
        squares.copy_(torch.stack([c.square().sum(-1) for c in x.chunk(self.parts, -1)], -1))
        self.folded += 1
        return True

    def linear(self, a, w, bias, out):
        if not isinstance(a, ScaledRows):
            return super().linear(a, w, bias, out)
        factor = (a.squares.sum(-1, keepdim=True) / a.rows.shape[1] + a.eps).rsqrt()
        out.copy_((a.rows.float() @ w.float().T * factor + (0 if bias is None else bias)).to(out.dtype))
        self.scaled_products += 1


def model_of(schedule=((0, False), (1, False)), final=None, make=lambda kind, params: PartSpec(kind, params)):
    """A decoder of two layers, its schedule entries (layer, adds the embedding again); `make` renames kinds."""
    rms = make("rmsnorm", {"size": D, "eps": EPS})
    attn = make("gqa_attention", {"hidden_size": D, "num_heads": 2, "num_kv_heads": 1, "head_dim": 16, "scale": 0.25, "window": 0, "position": "rope"})
    ffn = make("swiglu", {"hidden_size": D, "intermediate_size": 2 * D})
    layers = tuple(LayerSpec(f"m.{i}.", make("pre_norm", {}), attn, ffn, rms) for i in range(2))
    return DecoderModel(ModelSpec(
        architecture="toy_pending", hidden_size=D, vocab_size=V, embed_name="m.embed.weight", lm_head_name=None, tie_embeddings=True,
        final_norm=final or rms, final_norm_name="m.norm.weight", layers=layers,
        schedule=tuple(ScheduleEntry(layer, i, add_embedding=add) for i, (layer, add) in enumerate(schedule)),
        positions={"rope": make("rope", {"head_dim": 16, "theta": 100.0})}, max_position=64))


def bound(model, ops, seed=0):
    g = torch.Generator().manual_seed(seed)
    w = {name: 1 + 0.1 * torch.randn(p.shape, generator=g) if p.init == "ones" else torch.randn(p.shape, generator=g) * 0.3
         for name, p in model.expected_tensors().items() if not p.ignore and p.group is None}
    model.ops = ops
    return model.bind(w, ops, "float32", torch.device("cpu"), 64)


def logits(model):
    """Of two prompts in one step, then of a token more for each."""
    cache = CacheManager(model.cache_needs(), model.state_needs(), 4, 20, 2, 32, torch.float32, "cpu")
    runner = StepRunner(model, cache, max_rows=16, max_segments=2)
    out = [runner.run([Portion(r, ids, list(range(len(ids)))) for r, ids in enumerate(IDS)]).clone(),
           runner.run([Portion(r, [5 + r], [0]) for r in range(2)]).clone()]
    return torch.cat(out)


def same(got, want):
    assert torch.isfinite(got).all() and float((got - want).abs().max()) <= 2e-5 * float(want.abs().max())      # (float32 sums in another order)


OWN = {"gqa_attention": (MIXERS, GQAttention), "swiglu": (FEED_FORWARDS, SwiGLU), "rmsnorm": (NORMS, RMSNorm), "pre_norm": (BLOCKS, PreNormBlock),
       "rope": (POSITIONS, RotaryEncoding)}


@pytest.mark.parametrize("ops", [Plain, FoldingOps])
@pytest.mark.parametrize("kind", list(OWN))
def test_a_class_with_its_own_forward_is_run_by_it(kind, ops, monkeypatch):
    """A registered class that derives from a part of the package and brings its own `forward` (a position encoding: its own product
    with rotation and store), written for plain rows and pending terms."""
    table, base = OWN[kind]
    calls = []

    class Mixer(base):
        def forward(self, ctx, h, cache):
            calls.append(h.float().sum())      # (rows as a tensor)
            out = super().forward(ctx, h, cache)
            return out.mul_(0.5)

    class Ffn(base):
        def forward(self, ctx, h):
            calls.append(h.float().sum())
            return super().forward(ctx, h).mul_(0.5)

    class Norm(base):
        def forward(self, ctx, x, delta, rows=None, n_rows=None):
            calls.append(0)
            return super().forward(ctx, x, delta, rows, n_rows).mul_(0.5)

    class Block(base):
        def forward(self, ctx, x, delta, cache):
            calls.append(0)
            if delta is not None:
                delta = delta * 0.5
            x, delta = super().forward(ctx, x, delta, cache)
            return x, delta * 0.5

    class Position(base):
        def project_rotate_store(self, ctx, h, w, bias, q_out, cache, num_heads, num_kv_heads, head_dim):
            calls.append(h.float().sum())
            qkv = torch.empty(h.shape[0], w.shape[0])
            ctx.ops.linear(h, w, bias, qkv)
            self.rotate_and_store(ctx, qkv, q_out, cache, num_heads, num_kv_heads, head_dim)
            return True

    own = {"gqa_attention": Mixer, "swiglu": Ffn, "rmsnorm": Norm, "pre_norm": Block, "rope": Position}[kind]
    monkeypatch.setitem(table, "toy_own", own)
    got = logits(bound(model_of(make=lambda k, p: PartSpec("toy_own" if k == kind else k, p)), ops()))
    # two layers, two steps; a norm stands twice in a layer and once at the end (with rows folded into a product before it, the
    # rotation runs by itself: a fused one is optional)
    if kind != "rope" or ops is Plain:
        assert len(calls) == {"rmsnorm": 10}.get(kind, 4)
    plain = model_of()
    if kind == "pre_norm":      # the halved terms, by hand: a residual term counts 1/2, behind another block 1/4
        want = logits(bound(model_of(make=lambda k, p: PartSpec("toy_own" if k == kind else k, p)), Plain()))
    elif kind == "rope":
        want = logits(bound(plain, Plain()))
    else:
        m = bound(plain, Plain())
        for layer in m.layers:
            if kind == "gqa_attention":
                layer.mixer.wo = layer.mixer.wo * 0.5
            elif kind == "swiglu":
                layer.ffn.wd = layer.ffn.wd * 0.5
            else:
                layer.norm1.weight, layer.norm2.weight = layer.norm1.weight * 0.5, layer.norm2.weight * 0.5
        if kind == "rmsnorm":
            m.final_norm.weight = m.final_norm.weight * 0.5
        want = logits(m)
    same(got, want)


@pytest.mark.parametrize("ops", [Plain, FoldingOps])
@pytest.mark.parametrize("part", ["mixer", "ffn", "norm1", "norm2"])
def test_a_forward_replaced_on_the_object_is_run(part, ops):
    """What someone who watches a part does: the object's `forward` replaced by one that looks at its rows and results."""
    model, seen = bound(model_of(), ops()), []
    want = logits(bound(model_of(), Plain()))
    for layer in model.layers:
        p = getattr(layer, part)
        inner = p.forward

        def watch(ctx, first, *rest, inner=inner):
            out = inner(ctx, first, *rest)
            seen.append((float(first.float().sum()), float(out.float().sum())))
            return out
        p.forward = wraps(inner)(watch)
    same(logits(model), want)
    assert len(seen) == 4
    for layer in model.layers:      # and no longer, once it is taken away
        del getattr(layer, part).forward
    same(logits(model), want)
    assert len(seen) == 4 and not any(getattr(layer, part).own_forward for layer in model.layers)


@pytest.mark.parametrize("ops", [Plain, FoldingOps])
def test_a_block_that_is_watched_hands_its_terms_on(ops):
    """The stream behind every block, read off by the blocks' own `forward`."""
    model, plain, streams = bound(model_of(), ops()), bound(model_of(), Plain()), ([], [])
    for m, seen in zip((model, plain), streams):
        for layer in m.layers:
            def watch(ctx, x, delta, cache, inner=layer.forward, seen=seen):
                x, delta = inner(ctx, x, delta, cache)
                seen.append(x + delta)
                return x, delta
            layer.forward = watch
        out = logits(m)
    same(logits(model), out)
    for got, want in zip(*streams):
        same(got, want)


def test_who_takes_a_product():
    """Folded: every norm behind a sublayer but the last, which selects rows."""
    ops = FoldingOps()
    want = logits(bound(model_of(), Plain()))
    same(logits(bound(model_of(), ops)), want)
    assert ops.folded == 2 * 3 and ops.scaled_products == 2 * 3      # a step: norm2 of both layers, norm1 of the second


@pytest.mark.parametrize("schedule,folded", [
    (((0, False), (0, False), (1, False)), 5),             # a layer twice: every successor takes its product
    (((0, False), (1, False), (0, True)), 4),              # the embedding added behind layer 1, not behind layer 0
    (((0, False), (1, True), (0, False), (1, False)), 5),  # behind layer 0 once with and once without the embedding: never left
])
def test_products_of_layers_run_more_than_once(schedule, folded):
    ops = FoldingOps()
    want = logits(bound(model_of(schedule), Plain()))
    same(logits(bound(model_of(schedule), ops)), want)
    assert ops.folded == 2 * folded


def test_a_last_norm_that_takes_no_products():
    final = PartSpec("layernorm", {"size": D, "eps": EPS})

    class Ops(FoldingOps):
        def add_layernorm(self, x, delta, extra, weight, eps, h, rows=None, **options):
            y = x[rows.long()] + delta[rows.long()]
            h.copy_(torch.nn.functional.layer_norm(y, (D,), weight, None, eps).to(h.dtype))

    ops, plain = Ops(), Ops()
    plain.parts = 0
    want = logits(bound(model_of(final=final), plain))
    same(logits(bound(model_of(final=final), ops)), want)
    assert ops.folded == 6 and plain.folded == 0


def test_a_table_that_refuses_the_operands_gets_the_product_and_the_norm():
    class Refuses(FoldingOps):
        def linear_add_norm(self, *args):
            return False
    ops = Refuses()
    want = logits(bound(model_of(), Plain()))
    assert torch.equal(logits(bound(model_of(), ops)), want) and ops.scaled_products == 0


def test_a_pending_product_is_the_product():
    ops = Plain()
    a, w, b = torch.randn(3, 8), torch.randn(5, 8), torch.randn(5)

    class Ctx:
        pass
    ctx = Ctx()
    ctx.ops = ops
    from fusezap_core_b200.engine.step import Workspace
    ctx.ws = Workspace(torch.device("cpu"), 4)
    assert torch.equal(PendingProduct(a, w, b).resolve(ctx, None), a @ w.T + b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("in_place", [True, False])
def test_a_norm_weight_changed_after_loading(dtype, in_place):
    """Folded or not, a norm multiplies by the weight it has at the call, in the type it has."""
    out = []
    for ops in (Plain(), FoldingOps()):
        model = bound(model_of(), ops)
        norms = [n for layer in model.layers for n in (layer.norm1, layer.norm2)]
        for n in norms:
            n.bind({"weight": n.weight.to(dtype)}, ops)
        logits(model)
        for i, n in enumerate(norms):
            new = torch.linspace(0.5, 1.5 + i, D).to(dtype)
            if in_place:
                n.weight.copy_(new)
            else:
                n.weight = new
        out.append(logits(model))
    same(out[1], out[0])
