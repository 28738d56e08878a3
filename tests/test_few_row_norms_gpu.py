"""The norms of single-token steps (a thread four columns, everything asked for at once) against 64 bits, at the edges of the
sizes they take, beside the sizes the general kernels keep."""
import pytest
import torch

from camelid_b200.csrc import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"
# (rows, hidden): the smallest, a warp that is not whole, the largest, one beyond it, no whole groups of four, many rows
SIZES = [(1, 4), (3, 36), (8, 2048), (63, 1000), (2, 4096), (2, 4100), (5, 1022), (64, 256)]


def _rms(x, w=None, eps=1e-5):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w.double()


def _close(got, want, unit):
    """``unit``: half a unit in the last place of the output's type; beside it sums of squares and a few float roundings of
    terms of up to 5 or so, which may cancel (5 x 4 x 2^-23 < 2^-18)."""
    assert ((got.double() - want).abs() <= (unit + 2.0 ** -20) * want.abs() + 2.0 ** -18).all()


def _unit(dtype):
    return 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,hidden", SIZES)
def test_rmsnorm(rows, hidden, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows + hidden)
    x = torch.randn((rows + 2, hidden), generator=g, device=DEV)
    w, w2 = (torch.rand(hidden, generator=g, device=DEV).add(0.5).to(dtype) for _ in range(2))
    index = torch.arange(rows, device=DEV, dtype=torch.int32).flip(0) + 1
    out, out2 = (torch.empty((rows, hidden), dtype=dtype, device=DEV) for _ in range(2))
    ops.rmsnorm(x, w, 1e-5, out, index, None)
    _close(out, _rms(x.double(), w)[index.long()], _unit(dtype))
    ops.rmsnorm(x[:rows], w, 1e-5, out, None, None, w2, out2)
    _close(out, _rms(x[:rows].double(), w), _unit(dtype))
    _close(out2, _rms(x[:rows].double(), w2), _unit(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,hidden", SIZES)
def test_post_norm_add_and_combine(rows, hidden, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows + hidden)
    y, z, h = (torch.randn((rows, hidden), generator=g, device=DEV) for _ in range(3))
    w, nxt = (torch.rand(hidden, generator=g, device=DEV).add(0.5).to(dtype) for _ in range(2))
    bias = torch.randn(hidden, generator=g, device=DEV)
    for b in (None, bias):
        for then in (None, nxt):
            got, x = h.clone(), torch.empty((rows, hidden), dtype=dtype, device=DEV)
            ops.post_norm_add(y, b, w, 1e-5, 0.5, got, then, 1e-6, x)
            want = h.double() + 0.5 * _rms(y.double() + (b.double() if b is not None else 0.0), w)
            _close(got, want, 0.0)
            _close(x, _rms(got.double(), then, 1e-6) if then is not None else got.double(), _unit(dtype))
    got = h.clone()
    ops.norm_combine([(y, w), (z, nxt)], got, 1e-5, 0.25)
    _close(got, h.double() + 0.25 * (_rms(y.double(), w) + _rms(z.double(), nxt)), 0.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,hidden", SIZES)
def test_rmsnorm_shift(rows, hidden, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows + hidden)
    x = torch.randn((rows, hidden), generator=g, device=DEV)
    w, mix = torch.rand(hidden, generator=g, device=DEV).add(0.5).to(dtype), torch.rand(hidden, generator=g, device=DEV)
    state = torch.randn((rows + 3, 1, hidden), generator=g, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                      # noqa: E731
    slots, pos = [(2 * i + 1) % (rows + 3) if rows == 2 else rows + 2 - i for i in range(rows)], [i % 3 for i in range(rows)]
    kept, out = state.clone(), torch.empty((rows, hidden), dtype=dtype, device=DEV)
    ops.rmsnorm_shift(x, w, 1e-5, mix, kept, i32(list(range(rows))), i32(pos), i32(slots), out)
    _close(kept[slots, 0], _rms(x.double(), w), _unit(dtype))
    before = torch.where(torch.tensor(pos, device=DEV)[:, None] == 0, torch.zeros_like(x), state[slots, 0]).double()
    own = kept[slots, 0].double()
    want = own + (before - own) * mix.double()
    assert ((out.double() - want).abs() <= _unit(dtype) * want.abs() + 2.0 ** -22 * (own.abs() + before.abs())).all()
    rest = [s for s in range(rows + 3) if s not in slots]
    assert torch.equal(kept[rest], state[rest])


@pytest.mark.parametrize("splits", [1, 4, 8, 9, 16, 17])
@pytest.mark.parametrize("rows,hidden", [(1, 36), (8, 2048), (3, 4096), (2, 4100), (63, 64), (64, 64), (128, 64), (129, 64)])
def test_split_sums(rows, hidden, splits):
    """The rows' split sums are added and, where a norm settles the stream, written back."""
    g = torch.Generator(device=DEV).manual_seed(splits)
    part = torch.randn((splits, rows, hidden), generator=g, device=DEV) / splits ** 0.5
    h = torch.randn((rows, hidden), generator=g, device=DEV)
    w, mix = torch.rand(hidden, generator=g, device=DEV).add(0.5), torch.rand(hidden, generator=g, device=DEV)
    total = h.double() + part.double().sum(0)
    x, out = h.clone(), torch.empty((rows, hidden), device=DEV)
    ops.rmsnorm(x, w, 1e-5, out, None, part)
    _close(x, total, 0.0)
    _close(out, _rms(total, w), 0.0)
    x, index = h.clone(), torch.arange(rows, device=DEV, dtype=torch.int32).flip(0).contiguous()
    ops.rmsnorm(x, w, 1e-5, out, index, part)
    assert torch.equal(x, h)
    _close(out, _rms(total, w).flip(0), 0.0)
    x, state = h.clone(), torch.zeros((rows, 1, hidden), device=DEV)
    zero, own = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.arange(rows, dtype=torch.int32, device=DEV)
    ops.rmsnorm_shift(x, w, 1e-5, mix, state, own, zero, own, out, part)
    _close(x, total, 0.0)
    _close(state[:, 0], _rms(total, w), 0.0)
    x = h.clone()
    ops.post_norm_add(part, None, w, 1e-5, 0.5, x)
    _close(x, h.double() + 0.5 * _rms(part.double().sum(0), w), 0.0)


def test_rows_and_weights_of_the_kernel_before():
    """Rows that a kernel right before has chosen, and weights that it has written: without ``early`` a norm waits for them."""
    g = torch.Generator(device=DEV).manual_seed(0)
    rows, hidden, choices = 8, 256, 512
    x = torch.randn((choices, hidden), generator=g, device=DEV)
    w = torch.ones(hidden, device=DEV)
    ids, wts = torch.zeros(rows, dtype=torch.int32, device=DEV), torch.empty(rows, device=DEV)
    zero = torch.zeros(rows, dtype=torch.int32, device=DEV)
    own, mix = torch.arange(rows, dtype=torch.int32, device=DEV), torch.zeros(hidden, device=DEV)
    got, want = [], []
    for i in range(20):
        best = torch.randperm(choices, generator=torch.Generator().manual_seed(i))[:rows].to(DEV)
        logits = torch.randn((rows, choices), generator=g, device=DEV).scatter_(1, best[:, None], 9.0)
        state, h, out = torch.zeros((choices, 1, hidden), device=DEV), x[:rows].clone(), torch.empty((rows, hidden), device=DEV)
        torch.cuda.synchronize()
        ops.route_topk(logits, 1, True, False, ids, wts)
        ops.rmsnorm(x, w, 1e-5, out, ids)
        ops.route_topk(logits, 1, True, False, ids, wts)
        ops.rmsnorm_shift(x[:rows], torch.ones_like(w), 1e-5, mix, state, own, zero, ids, torch.empty_like(out))
        ops.scale_(w, 2.0)
        ops.post_norm_add(x[:rows], None, w, 1e-5, 1.0, h)
        ops.scale_(w, 0.5)
        ops.norm_combine([(x[:rows], w)], h, 1e-5, 1.0)
        got.append((out, state[best, 0], h))
        n = _rms(x.double())
        want.append((n[best], n[:rows], x[:rows].double() + 3 * n[:rows]))
    for a, b in zip(got, want):
        for y, z in zip(a, b):
            _close(y, z, 2.0 ** -22)


@pytest.mark.parametrize("key_dim,value_dim", [(0, 8), (8, 0), (0, 0)])
def test_heads_without_channels(key_dim, value_dim):
    """Heads of no channels have nothing that could be read: the others' numbers, and no access in front of an array."""
    G, H, rows, guard = 1, 2, 2, 8
    channels = 2 * G * key_dim + H * value_dim
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)                      # noqa: E731
    g = torch.Generator(device=DEV).manual_seed(0)
    mem = torch.randn((5, 64 * guard), generator=g, device=DEV)
    proj, w, out = mem[0][guard:guard + rows * channels].view(rows, channels), mem[1][guard:guard + channels * 4], mem[2][guard:guard + rows * channels]
    state = mem[3][guard:guard + rows * 3 * channels]
    at = lambda t, i: mem[i].data_ptr() + 4 * guard                                     # noqa: E731
    before, x, taps = mem.clone(), proj.double().clone(), w.double().view(channels, 4).clone()
    ints = [i32([0, 1]), i32([0, 0]), i32([0, 1]), i32([0, 1])]
    code = ops._fn("recurrence", "cml_conv_unit")(at(proj, 0), channels, at(w, 1), at(state, 3), 1, *(t.data_ptr() for t in ints), at(out, 2), rows, G, H,
                                                  key_dim, value_dim, 4, 0.5, None, 0, None, None, None, 1, 0, ops._stream())
    assert code == 0
    y = torch.nn.functional.silu(x * taps[:, 3])                # (first tokens: the taps before them see nothing)
    q, v = y[:, :2 * G * key_dim].view(rows, 2 * G, key_dim), y[:, 2 * G * key_dim:]
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * torch.tensor([0.5, 1.0], device=DEV)[:, None]
    want = torch.cat([q.flatten(1), v], 1).flatten()
    assert ((out.double() - want).abs() <= 1e-5).all()
    assert torch.equal(mem[2][:guard], before[2][:guard]) and torch.equal(mem[2][guard + rows * channels:], before[2][guard + rows * channels:])
    kept = mem[4].clone()
    code = ops._fn("recurrence", "cml_head_norm_gate")(at(proj, 0), 0, 0, at(w, 1), 0, at(state, 3), 0, 0, at(out, 4), 0, ops.dtype_code(torch.float32), rows,
                                                       H, 0, 1e-6, 0, ops._stream())
    assert code == 0 and torch.equal(mem[4], kept)


def test_rows_without_columns():
    """Nothing to norm is no error."""
    x, w = torch.empty((2, 0), device=DEV), torch.empty(0, device=DEV)
    ops.rmsnorm(x, w, 1e-5, torch.empty_like(x))
