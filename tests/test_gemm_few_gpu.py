"""The product of few rows (gemm_few.cu) against the same sums in 64 bits: edges of its tiles of 16 features and stages of
512 columns, K in one and split, strided operands, every epilogue."""
import pytest
import torch

from camelid_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
# (rows, features, columns): one lane's piece of K, K's last 64 and 512 cut short, one tile, more tiles than SMs, more
# stages than the ring holds, K of two to seven splits of which the last has less to do
SIZES = [(1, 16, 8), (1, 1, 512), (3, 17, 520), (8, 2048, 2048), (6, 40, 1000), (8, 2400, 1536), (5, 7000, 24), (8, 96, 5128), (2, 31, 8192),
         (4, 4744, 3080), (1, 2400, 2056), (3, 50, 4160), (8, 7000, 4104), (5, 2400, 9216),
         (7, 1300, 2568), (8, 40, 14336)]


def _operands(rows, n, k, seed=0, strided=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    pad = 24 if strided else 0
    x = torch.randn((rows, k + pad), generator=g, device=DEV).to(torch.bfloat16)[:, :k]
    w = (torch.randn((n, k + pad), generator=g, device=DEV) / k ** 0.5).to(torch.bfloat16)[:, :k]
    return x, w, torch.zeros(1, dtype=torch.int32, device=DEV)


def _bound(x, w):
    """What float sums of K products may lie off: the products are exact, each of K adds rounds (or cuts off) a partial sum."""
    return x.shape[1] * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("rows,n,k", SIZES)
def test_sums(rows, n, k, strided):
    x, w, err = _operands(rows, n, k, strided=strided)
    want, bound = x.double() @ w.double().T, _bound(x, w)
    splits = ops.few_splits(k)
    wide = torch.full((splits, rows, n + 3), 7.0, device=DEV)
    ops.gemm_few(x, w, wide[..., :n], ops.FEW_F32, err)
    assert ((wide[..., :n].double().sum(0) - want).abs() <= bound).all() and (wide[..., n:] == 7).all() and int(err) == 0
    assert splits == -(-k // 2048)
    if splits > 1:
        return                                                  # (the other epilogues take whole sums)
    add = torch.randn((rows, n), device=DEV)
    got = add.clone()
    ops.gemm_few(x, w, got, ops.FEW_ADD, err)
    assert ((got.double() - (want + add.double())).abs() <= bound + 2.0 ** -23 * (want + add.double()).abs()).all()
    bias = torch.randn(n, device=DEV)
    for act, f in ((ops.ACT_NONE, lambda z: z), (ops.ACT_RELU_SQUARED, lambda z: torch.relu(z) ** 2),
                   (ops.ACT_GELU_TANH, lambda z: torch.nn.functional.gelu(z, approximate="tanh")), (ops.ACT_GELU_ERF, torch.nn.functional.gelu)):
        half = torch.empty((rows, n), dtype=torch.bfloat16, device=DEV)
        ops.gemm_few(x, w, half, ops.FEW_BF16, err, bias=bias, act=act)
        ref = f(want + bias.double())
        slope = 2 * torch.relu(want + bias.double()) + 2        # how much an error of the sum grows (at most) through the activation
        assert ((half.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + slope * (bound + 2.0 ** -22 * (want.abs() + bias.double().abs() + 1))).all(), act


@pytest.mark.parametrize("rows,inter,k", [(1, 16, 8), (8, 1024, 512), (7, 2416, 1000), (2, 1200, 2048), (8, 2512, 1600)])
def test_gated(rows, inter, k):
    from camelid_b200.parts.linear import pack_gate_up
    x, w, err = _operands(rows, 2 * inter, k, seed=1)
    packed = pack_gate_up(w[:inter], w[inter:], 16)
    g, u = x.double() @ w[:inter].double().T, x.double() @ w[inter:].double().T
    out = torch.empty((rows, inter), dtype=torch.bfloat16, device=DEV)
    for gate in (None, ops.GateAct(1.702, 1.0, 1.0)):
        ops.gemm_few(x, packed, out, ops.FEW_GATED, err, gate=gate)
        a, lim, shift = gate or ops.SILU_GATE
        gc, uc = g.clamp(max=lim), u.clamp(-lim, lim)
        ref = gc * torch.sigmoid(a * gc) * (uc + shift)
        # the activation's fast exponential and division: some units in the last place of float
        assert ((out.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * (1 + gc.abs()) * (1 + uc.abs())).all()


@pytest.mark.parametrize("weight", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n,k,next_n", [(1, 2048, 512, 64), (8, 40, 1024, 33), (7, 2040, 64, 520), (4, 1600, 1544, 16), (3, 96, 2048, 2400),
                                             (8, 2304, 2048, 40), (5, 4096, 264, 2400)])      # (the last two: the reader's K comes in shares)
def test_add_norm_and_the_scale_left_undone(rows, n, k, next_n, weight):
    """The residual add with the norm behind it, then a product of the rows that still lack their scale."""
    x, w, err = _operands(rows, n, k, seed=2)
    h = torch.randn((rows, n), device=DEV)
    nw = (1 + torch.rand(n, device=DEV)).to(weight)
    want = h.double() + x.double() @ w.double().T
    xo = torch.empty((rows, n), dtype=torch.bfloat16, device=DEV)
    sumsq = torch.empty(((n + 15) // 16, rows), device=DEV)
    ops.gemm_few(x, w, h, ops.FEW_ADD_NORM, err, norm=(nw, xo, sumsq))
    bound = _bound(x, w) + 2.0 ** -22 * want.abs()
    assert ((h.double() - want).abs() <= bound).all()
    assert torch.equal(xo, (h * nw.float()).to(torch.bfloat16))
    sums = torch.nn.functional.pad(h.double() ** 2, (0, -n % 16)).view(rows, -1, 16).sum(-1).T
    assert ((sumsq.double() - sums).abs() <= 2.0 ** -20 * sums).all()
    w2 = (torch.randn((next_n, n), device=DEV) / n ** 0.5).to(torch.bfloat16)
    scale = ops.RowScale(sumsq, n, 1e-5)
    out = torch.empty((ops.few_splits(n), rows, next_n), device=DEV)
    ops.gemm_few(xo, w2, out, ops.FEW_F32, err, row_scale=scale)
    out = out.sum(0)
    rs = torch.rsqrt((h.double() ** 2).mean(-1, keepdim=True) + 1e-5)
    ref = rs * (xo.double() @ w2.double().T)
    assert ((out.double() - ref).abs() <= rs * _bound(xo, w2) + 2.0 ** -20 * ref.abs()).all() and int(err) == 0
    # or scaled in place, from the same sums of squares per 16 columns
    done = xo.clone()
    ops.scale_rows(done, scale)
    assert ((done.double() - rs * xo.double()).abs() <= (2.0 ** -8 + 2.0 ** -20) * (rs * xo.double()).abs()).all()


def test_rows_that_are_not_finite_stay_apart():
    """What shared memory held before, the columns beyond K and a row with infinities touch no other row's sums."""
    x, w, err = _operands(6, 48, 1016, seed=3)                  # (six rows of eight, the last 64 columns cut short)
    out = torch.empty((6, 48), device=DEV)
    ops.gemm_few(x, w, out, ops.FEW_F32, err)
    bad = x.clone()
    bad[2] = float("inf")
    bad[4, 7] = float("nan")
    got = torch.empty_like(out)
    ops.gemm_few(bad, w, got, ops.FEW_F32, err)
    keep = [0, 1, 3, 5]
    assert torch.equal(got[keep], out[keep]) and not torch.isfinite(got[4]).any()


@pytest.mark.parametrize("rows,top,experts,n,k", [(1, 1, 3, 32, 8), (2, 2, 16, 1024, 1024), (8, 2, 5, 96, 520), (4, 4, 7, 2080, 2048), (5, 3, 4, 64, 1000), (8, 8, 9, 96, 264)])
def test_routed(rows, top, experts, n, k):
    """A matrix of its own for every (row, choice) pair; choices beyond the experts leave their rows alone."""
    from camelid_b200.parts.linear import pack_gate_up
    x, w, err = _operands(rows, experts * n, k, seed=4)
    w = w.view(experts, n, k)
    ids = torch.randint(0, experts + 1, (rows * top,), generator=torch.Generator().manual_seed(rows)).to(torch.int32)
    ids[0] = experts - 1
    out = torch.full((rows * top, n), 7.0, device=DEV)
    ops.gemm_few_experts(x, top, w, out, ops.FEW_F32, ids.to(DEV), err)
    packed = torch.stack([pack_gate_up(m[:n // 2], m[n // 2:], 16) for m in w])
    act = torch.full((rows * top, n // 2), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.gemm_few_experts(x, top, packed, act, ops.FEW_GATED, ids.to(DEV), err)
    for i, e in enumerate(ids.tolist()):
        if e == experts:
            assert (out[i] == 7).all() and (act[i] == 7).all()
            continue
        row = x[i // top:i // top + 1]
        want = (row.double() @ w[e].double().T)[0]
        assert ((out[i].double() - want).abs() <= _bound(row, w[e])[0]).all()
        g, u = want[:n // 2], want[n // 2:]
        ref = g * torch.sigmoid(g) * u
        assert ((act[i].double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-4 * (1 + g.abs()) * (1 + u.abs())).all()
    assert int(err) == 0


@pytest.mark.parametrize("name", ["llama", "llama of 5120", "fomatar", "zulozen", "kizezen", "ramopel", "zabunex"])
def test_decoders_on_either_path(name):
    """Steps of few rows (a short prompt, single tokens) on this kernel and on the products of more rows."""
    import camelid_b200
    from camelid_b200 import KernelOptions, StepEntry, benchmark
    wide = {"hidden_size": 5120, "num_hidden_layers": 3, "intermediate_size": 1024, "vocab_size": 3000}      # norms of rows the register kernel does not take
    cfg = {**benchmark.llama_config_like("small"), **(wide if "of" in name else {})} if name.startswith("llama") else benchmark.zulozen_config_like_kizezen("small") if name == "zulozen" \
        else getattr(benchmark, name + "_config_for")("small")
    got = []
    for few in (True, False):
        lm = camelid_b200.from_random(cfg, seed=3, dtype="bfloat16", options=KernelOptions(few_rows=few))
        cache = lm.new_cache(256, max_slots=3)
        slots, rows = [cache.alloc_slot() for _ in range(3)], []
        for i, s in enumerate(slots):
            rows.append(lm.step(cache, [StepEntry(s, [11 * i + j for j in range(3 + 2 * i)], [2 + 2 * i])]).clone())
        for t in range(4):
            rows.append(lm.step(cache, [StepEntry(s, [5 + t + i], [0]) for i, s in enumerate(slots)]).clone())
        got.append(torch.cat(rows).double())
        del lm, cache
    # every kernel rounds the rows it hands on to one part in 256, in another order of sums on either path
    assert (got[0] - got[1]).norm() <= 3e-2 * got[1].norm()


# (width, heads of 16 or 64, feed-forward): K of gate/up beyond what one block sums; no whole groups of 8; interleaved in one group
@pytest.mark.parametrize("width,heads,dim,ff", [(2560, 32, 64, 1024), (100, 4, 16, 160), (512, 4, 64, 1000)])
def test_rows_between_products_are_rounded_once(monkeypatch, width, heads, dim, ff):
    """Where the gate/up product cannot scale its sums, the norm in front of it is whole: nothing scales rows that are in bfloat16 already."""
    import camelid_b200
    from camelid_b200 import StepEntry, benchmark
    cfg = {**benchmark.llama_config_like("small"), "hidden_size": width, "num_hidden_layers": 2, "num_attention_heads": heads,
           "num_key_value_heads": 2, "head_dim": dim, "intermediate_size": ff}
    lm = camelid_b200.from_random(cfg, seed=3, dtype="bfloat16")
    monkeypatch.setattr(ops, "scale_rows", lambda *a: pytest.fail("rows in bfloat16 are scaled, and so rounded, a second time"))
    cache = lm.new_cache(1024, max_slots=2)
    slots = [cache.alloc_slot() for _ in range(2)]
    for n in (3, 300, 1):                                       # few rows, many rows, single tokens
        lm.step(cache, [StepEntry(s, list(range(n)), [n - 1]) for s in slots])


def test_routed_experts_that_load_their_matrices_themselves():
    """A derived part whose ``load`` knows nothing of the unsorted form runs sorted, as it did."""
    from camelid_b200.engine.context import StepContext, Workspace
    from camelid_b200.parts.experts import RoutedExperts
    from camelid_b200.weights import random_tensors

    class Own(RoutedExperts):
        def load(self, tensors, device, dtype):
            super().load(tensors, device, dtype)
            del self.pair_order

    got = []
    for cls in (RoutedExperts, Own):
        part = cls({"hidden_size": 64, "expert_size": 48, "experts": 4, "top": 2}, "m.")
        part.load(random_tensors(part.tensor_specs(), 0, torch.bfloat16), DEV, torch.bfloat16)
        x = torch.randn((3, 64), generator=torch.Generator().manual_seed(0)).to(torch.bfloat16).to(DEV)
        ctx = StepContext.for_step(cache=None, workspace=Workspace(torch.device(DEV)), dtype=torch.bfloat16, device=DEV, slots=[0], starts=[0],
                                   tokens=[[0] * 3], want=[[]])
        h = torch.zeros((3, 64), device=DEV)
        part.forward(ctx, x, h)
        got.append(h.double())
    # rows of 48 activations rounded to bfloat16, sums in another order
    assert (got[0] - got[1]).norm() <= 1e-2 * got[0].norm() > 0


@pytest.mark.parametrize("name", ["llama", "kizezen"])
@pytest.mark.parametrize("rows", [5, 300])
def test_norms_inside_the_products_or_on_their_own(name, rows):
    """The weight half of a norm in the product before it and its scale behind the product after it, against norms of their own: the
    gated feed-forward and grouped-query attention, and (kizezen) the dense feed-forward, window and latent attention and retention."""
    import camelid_b200
    from camelid_b200 import KernelOptions, StepEntry, benchmark
    cfg = benchmark.llama_config_like("small") if name == "llama" else benchmark.kizezen_config_for("small")
    got, launches = [], []
    for fuse in (True, False):
        lm = camelid_b200.from_random(cfg, seed=3, dtype="bfloat16", options=KernelOptions(fuse_norm=fuse))
        cache = lm.new_cache(1024, max_slots=1)
        before = ops.launch_count()
        got.append(lm.step(cache, [StepEntry(cache.alloc_slot(), [(7 * i) % 251 for i in range(rows)], list(range(rows)))]).double())
        launches.append(ops.launch_count() - before)
        takers = {type(p).__name__ for b in lm.model.blocks for p in (b.mixer, b.ffn) if p is not None and p.accepts_row_scale}
        del lm, cache
    assert takers == ({"GroupedQueryAttention", "SwiGLU"} if name == "llama" else {"DenseFeedForward", "LatentAttention", "Retention", "WindowAttention"})
    assert launches[0] < launches[1]                            # (every fused norm is a launch less)
    # a row's bfloat16 rounding falls before its scale or behind it
    assert (got[0] - got[1]).norm() <= 3e-2 * got[1].norm()
