"""The Gamilorn design on the GPU against the plain implementation of ``tests/plain_gamilorn.py``:
each new kernel alone (inputs made so that one far key, a key just inside or just outside the
window or the kept first keys, a page's border or a lost state would show), then whole models
through ``bin/trace_run`` (whole prompts, the last tokens one by one over more tokens than the
windows are long, portions down to two tokens, mixed batches in a pool so small that pages
and state slots are used again), in float32 and bfloat16, and greedy generation through
``Engine.generate``."""

import math
from types import SimpleNamespace

import pytest
import torch

from tests import gamilorn_util as gu
from tests import plain_gamilorn as pg
from tests import replay_util as ru

pytestmark = pytest.mark.gpu

DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}


@pytest.fixture(scope="module")
def model_dirs(tmp_path_factory):
    return {name: gu.write_tiny(name, tmp_path_factory.mktemp(f"gamilorn_{name}")) for name in gu.CONFIGS}


def close(got, want, dtype, what, f32=2e-5, bf16=1.2e-2):
    got, want = got.double().cpu(), want.double().cpu()
    scale = float(want.abs().max())
    err = float((got - want).abs().max())
    bound = (f32 if dtype == "float32" else bf16) * max(scale, 1e-6)
    assert err <= bound, f"{what} ({dtype}): abs diff {err:.4g} exceeds {bound:.4g} (scale {scale:.4g})"


# ---- small kernels -------------------------------------------------------------------------------

@pytest.mark.parametrize("dtype", list(DTYPES))
def test_stream_kernels_alone(dtype):
    from deterministic_inference_b200.kernels import ops
    dt, dev = DTYPES[dtype], "cuda"
    g = torch.Generator().manual_seed(1)
    rows, width = 37, 136
    ids = torch.randint(0, 50, (rows,), generator=g, dtype=torch.int32)
    pos = torch.randint(0, 70, (rows,), generator=g, dtype=torch.int32)
    table, ptable = (torch.randn(n, width, generator=g).to(dt) for n in (50, 70))
    x = ops.embedding_positions(ids.to(dev), pos.to(dev), table.to(dev), ptable.to(dev))
    assert x.dtype == torch.float32
    want = table.double()[ids.long()] + ptable.double()[pos.long()]
    close(x, want, "float32", "embedding + position")

    # the stream takes two scaled terms (a stored tensor and split partial products) in float32
    w = torch.randn(width, generator=g) * 0.1
    a = torch.randn(rows, width, generator=g).to(dt)
    parts = torch.randn(3, rows, width, generator=g)
    stream = x.clone()
    y = ops.stream_rms_norm(stream, (1.0 + w).to(dev), 3e-5, dt,
                            add=ops.WeightedSum([(1.2, a.to(dev)), (0.7, ops.SplitSum(parts.to(dev), torch.float32))]))
    total = want + 1.2 * a.double() + 0.7 * parts.double().sum(0)
    close(stream, total, "float32", "stream after the addition")
    close(y, pg.zero_centred_norm(total, w.double(), 3e-5), dtype, "norm of the stream")
    close(ops.stream_rms_norm(stream, (1.0 + w).to(dev), 3e-5, dt), pg.zero_centred_norm(total, w.double(), 3e-5),
          dtype, "norm alone")

    z = torch.randn(rows, width, generator=g) * 3
    p, q = torch.tensor(0.3), torch.tensor(-0.8)
    sp = torch.nn.functional.softplus
    got = ops.xielu(z.to(dev), float(sp(p)), float(0.5 + sp(q)), dt)
    close(got, pg.xielu(z.double(), p.double(), q.double()), dtype, "xielu")
    logits = torch.randn(5, 77, generator=g) * 20
    close(ops.softcap_(logits.clone().to(dev), 11.0), pg.softcap(logits.double(), 11.0), "float32", "soft cap")


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("rows, width, splits", [(3, 4, 1), (5, 132, 3), (2048, 12, 1), (700, 2052, 1), (148, 256, 1),
                                                 (400, 3072, 2)])
def test_elements_by_fours_are_those_one_by_one(dtype, rows, width, splits):
    """The element-wise kernels on memory that allows vectors of four and on the same values one element further on,
    which does not: the same bits."""
    from deterministic_inference_b200.kernels import ops
    dt, dev = DTYPES[dtype], "cuda"
    g = torch.Generator(device=dev).manual_seed(width)

    def both(f, kind=torch.float32):
        x = (3 * torch.randn(splits, rows, width, generator=g, device=dev)).to(kind)
        there = torch.empty(x.numel() + 1, dtype=kind, device=dev)[1:].view(x.shape).copy_(x)
        source = lambda t: ops.SplitSum(t, torch.float32) if splits > 1 else t[0]
        assert torch.equal(f(source(x)), f(source(there)))

    both(lambda z: ops.xielu(z, 0.7, 1.3, dt))
    both(lambda z: ops.squared_relu(z, dt))
    if splits == 1:
        both(lambda z: ops.softcap_(z, 11.0))
        both(lambda z: ops.scale_(z, 0.3))
        both(lambda z: ops.xielu(z, 0.7, 1.3, dt), torch.bfloat16)
    dim = width // 4
    bias = torch.randn(width, generator=g, device=dev)
    slots = torch.randperm(rows, device=dev).int()
    caches = []

    def split_heads(qkv):
        caches.append(torch.zeros(-(-rows // 16), 16 * 3 * dim, dtype=dt, device=dev))
        return ops.qkv_bias_cache(qkv, bias, 1, 1, dim, 2 * dim, caches[-1], slots, 16, dt)

    both(split_heads)
    assert torch.equal(caches[0], caches[1])


# ---- attention without a softmax ---------------------------------------------------------------------

def paged(n_tokens_per_seq, page, generator):
    """Block tables over shuffled pages for sequences of the given lengths."""
    need = [-(-n // page) for n in n_tokens_per_seq]
    perm = (torch.randperm(sum(need), generator=generator) + 1).tolist()
    bt = torch.zeros(len(need), max(need), dtype=torch.int32)
    for b, n in enumerate(need):
        for i in range(n):
            bt[b, i] = perm.pop()
    return bt, sum(need) + 1


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("heads, kv_heads, dim, vdim, page, window, keep", [
    (6, 2, 24, 40, 16, 37, 5),      # values wider than keys, a window that ends inside a page
    (4, 4, 16, 16, 8, None, 0),     # no window, one query head per key head
    (8, 1, 32, 16, 16, 7, 19),      # more kept keys than the window is long
    (2, 1, 128, 64, 32, 64, 0),     # no kept keys, a window of two pages
    (6, 2, 32, 48, 16, 37, 70),     # three heads to a group; kept keys beyond the first key tile
    (5, 5, 64, 192, 16, 100, 3),    # wide values
])
def test_sigmoid_attention_alone(dtype, heads, kv_heads, dim, vdim, page, window, keep):
    from deterministic_inference_b200.kernels import ops
    dt, dev = DTYPES[dtype], "cuda"
    g = torch.Generator().manual_seed(heads * 100 + dim)
    n, n2 = 150, 45
    scale = 0.9 / math.sqrt(dim)
    rnd = pg.as_stored_bf16 if dtype == "bfloat16" else (lambda t: t)
    seqs = []
    for length in (n, n2):
        q = rnd(torch.randn(length, heads, dim, generator=g))
        k = rnd(torch.randn(length, kv_heads, dim, generator=g))
        v = rnd(torch.randn(length, kv_heads, vdim, generator=g))
        seqs.append([q, k, v])
    # keys whose weight is 1 against every query of the last tokens, with values that show: just
    # inside and just outside the window of the last position, the last kept key and the first
    # that is not kept, and a far key
    q, k, v = seqs[0]
    last = n - 1
    spikes = [0, n // 2]
    if window:
        spikes += [last - window + 1, last - window]
    if keep:
        spikes += [keep - 1, keep]
    q[last - 3:] = rnd(q[last - 3:] * 0.1 + 4.0 / math.sqrt(dim))
    for j in spikes:
        k[j] = rnd(torch.full_like(k[j], 3.0 / scale / math.sqrt(dim)))
        v[j] = rnd(v[j] + 50.0 * (1 + spikes.index(j)))
    bias = torch.randn(heads * dim + kv_heads * (dim + vdim), generator=g)
    head_bias = torch.randn(heads, generator=g) - 1.0
    bt, pages = paged([n, n2], page, g)
    cache = torch.zeros(pages, kv_heads * page * (dim + vdim), dtype=dt, device=dev)
    want = [pg.sigmoid_window_attention(q.double(), k.double(), v.double(), scale, head_bias.double(),
                                        window or 10 ** 9, keep) for q, k, v in seqs]

    # steps: a long portion of the first sequence alone; then portions of both; then single tokens
    steps = [[(0, 0, 90)], [(0, 90, 2), (1, 0, 31)], [(1, 31, 1), (0, 92, 13)], [(1, 32, 13), (0, 105, 41)]]
    steps += [[(0, p, 1)] for p in range(146, n)]
    got = [torch.zeros(n, heads, vdim, dtype=torch.float64), torch.zeros(n2, heads, vdim, dtype=torch.float64)]
    q_stored = torch.zeros(n, heads, dim, dtype=dt, device=dev)      # the first sequence's q as the kernel left it
    for entries in steps:
        rows, seq_of, pos_of, slots = [], [], [], []
        for b, (s, start, count) in enumerate(entries):
            qq, kk, vv = seqs[s]
            rows.append(torch.cat([qq[start:start + count].reshape(count, -1), kk[start:start + count].reshape(count, -1),
                                   vv[start:start + count].reshape(count, -1)], dim=1))
            for p in range(start, start + count):
                seq_of.append(b)
                pos_of.append(p)
                slots.append(int(bt[s, p // page]) * page + p % page)
        x = torch.cat(rows) - bias                  # the kernel adds the bias back
        meta = SimpleNamespace(block_table=bt[[s for s, _, _ in entries]].contiguous().to(dev),
                               token_seq=torch.tensor(seq_of, dtype=torch.int32, device=dev),
                               positions=torch.tensor(pos_of, dtype=torch.int32, device=dev),
                               seq_lens=torch.tensor([st + c for _, st, c in entries], dtype=torch.int32, device=dev),
                               q_lens=[c for _, _, c in entries], kv_lens=[st + c for _, st, c in entries],
                               scratch={}, num_decode=sum(1 for _, _, c in entries if c == 1))
        qd = ops.qkv_bias_cache(x.to(dev), bias.to(dev), heads, kv_heads, dim, vdim, cache,
                                torch.tensor(slots, dtype=torch.int32, device=dev), page, dt)
        out = ops.sigmoid_attention(qd, cache, meta, scale, head_bias.to(dev), vdim, page, window, keep).cpu()
        at = 0
        for s, start, count in entries:
            got[s][start:start + count] = out[at:at + count].double()
            if s == 0:
                q_stored[start:start + count] = qd[at:at + count]
            at += count
    for s in (0, 1):
        close(got[s], want[s], dtype, f"attention of sequence {s}", f32=3e-5, bf16=8e-3)
    # the same rows in one step: a row's bits do not depend on how the sequence was cut
    meta = SimpleNamespace(block_table=bt[:1].contiguous().to(dev), token_seq=torch.zeros(n, dtype=torch.int32, device=dev),
                           positions=torch.arange(n, dtype=torch.int32, device=dev),
                           seq_lens=torch.tensor([n], dtype=torch.int32, device=dev), q_lens=[n], kv_lens=[n],
                           scratch={}, num_decode=0)
    whole = ops.sigmoid_attention(q_stored, cache, meta, scale, head_bias.to(dev), vdim, page, window, keep)
    # (tokens that came alone ran on the kernel form for decoded tokens, which associates a
    # row's sum over its keys differently: a rounding apart at most)
    cut = 146 if dtype == "bfloat16" else n
    assert torch.equal(whole.cpu().double()[:cut], got[0][:cut]), "a row's bits changed with the cutting"
    if cut < n:
        close(whole[cut:], got[0][cut:], dtype, "tokens alone against the same tokens in a prompt", bf16=4e-3)
    # the spikes did show: a wrong edge would move the last row by about 50
    assert float(want[0][last].abs().max()) > 50


@pytest.mark.parametrize("heads, kv_heads, page, window, keep, lens", [
    (4, 2, 16, 100, 5, (300, 129)),        # a window within a tile of 128 keys, kept keys in the first
    (2, 2, 128, None, 0, (257, 64)),       # one head a group, a page a tile
    (8, 1, 8, 130, 140, (500, 2)),         # a window beyond a tile, kept keys beyond one; groups of 8
    (4, 1, 32, 256, 0, (640, 33)),
])
def test_sigmoid_attention_of_128(heads, kv_heads, page, window, keep, lens):
    """Keys and values of 128 (the tcgen05 form for prompt portions): against 64 bits at whole and ragged tiles; a row's
    bits do not depend on the portion it comes in; what a page holds past a sequence's end, not a number here, does
    not reach a row."""
    from deterministic_inference_b200.kernels import ops
    dim, dev = 128, "cuda"
    g = torch.Generator().manual_seed(heads + page)
    scale = 0.9 / math.sqrt(dim)
    rnd = lambda *s: pg.as_stored_bf16(torch.randn(*s, generator=g))
    seqs = [(rnd(n, heads, dim), rnd(n, kv_heads, dim), rnd(n, kv_heads, dim)) for n in lens]
    head_bias = torch.randn(heads, generator=g) - 1.0
    bt, pages = paged(list(lens), page, g)
    cache = torch.full((pages, 2, kv_heads, page, dim), float("nan"), dtype=torch.bfloat16)
    for b, (_, k, v) in enumerate(seqs):
        for p in range(lens[b]):
            cache[int(bt[b, p // page]), 0, :, p % page] = k[p].bfloat16()
            cache[int(bt[b, p // page]), 1, :, p % page] = v[p].bfloat16()
    cache = cache.view(pages, -1).to(dev)

    def run(entries):
        rows, seq_of, pos_of = [], [], []
        for i, (b, start, count) in enumerate(entries):
            rows.append(seqs[b][0][start:start + count])
            seq_of += [i] * count
            pos_of += range(start, start + count)
        i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=dev)
        meta = SimpleNamespace(block_table=bt[[b for b, _, _ in entries]].contiguous().to(dev), token_seq=i32(seq_of),
                               positions=i32(pos_of), seq_lens=i32([s + c for _, s, c in entries]),
                               q_lens=[c for _, _, c in entries], kv_lens=[s + c for _, s, c in entries], scratch={},
                               num_decode=0)
        out = ops.sigmoid_attention(torch.cat(rows).bfloat16().to(dev), cache, meta, scale, head_bias.to(dev), dim, page,
                                    window, keep).cpu()
        return list(out.split([c for _, _, c in entries]))

    whole = run([(0, 0, lens[0]), (1, 0, lens[1])])
    for b, (q, k, v) in enumerate(seqs):
        want = pg.sigmoid_window_attention(q.double(), k.double(), v.double(), scale, head_bias.double(),
                                           window or 10 ** 9, keep)
        close(whole[b].double(), want, "bfloat16", f"attention of sequence {b}", bf16=8e-3)
    cut = lens[0] // 2 + 3
    assert torch.equal(run([(1, 0, lens[1]), (0, cut, lens[0] - cut)])[1], whole[0][cut:])
    assert torch.equal(run([(0, 0, 2)])[0], whole[0][:2])
    ops.check_kernel_status()


# ---- the delta-rule recurrence -----------------------------------------------------------------------

@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("heads, dim, rank", [(3, 16, 4), (2, 40, 8), (2, 64, 16), (1, 128, 5), (1, 200, 2)])
def test_delta_rule_alone(dtype, heads, dim, rank):
    from deterministic_inference_b200.kernels import ops
    dt, dev = DTYPES[dtype], "cuda"
    g = torch.Generator().manual_seed(heads * 1000 + dim)
    hd = heads * dim
    lens = (70, 23)
    eps, key_eps, decay_scale = 2e-5, 1e-6, math.exp(-0.5)
    w2 = pg.as_stored_bf16(torch.randn(hd, rank, generator=g))
    w0, a_bias = torch.randn(hd, generator=g) - 3.0, torch.randn(hd, generator=g)       # slow decays: w near 1
    norm_w = 1.0 + 0.1 * torch.randn(hd, generator=g)
    projs, want = [], []
    for n in lens:
        proj = torch.randn(n, 5 * hd + rank, generator=g)
        # the first key comes back as the last query: what the state kept of token 0 shows at the end
        proj[-1, :hd] = 3.0 * proj[0, hd:2 * hd]
        projs.append(proj)
        p = proj.double()
        shape = (n, heads, dim)
        r, k, v, gate = (p[:, i * hd:(i + 1) * hd] for i in range(4))
        rate = torch.sigmoid(p[:, 4 * hd:5 * hd] + a_bias.double()).view(shape)
        decay = pg.decay_of(p[:, 5 * hd:], torch.eye(rank, dtype=torch.float64), w2.double(), w0.double()).view(shape)
        o, last = pg.delta_rule(r.reshape(shape), k.reshape(shape), v.reshape(shape), decay, rate)
        want.append((pg.unit_rms(o, eps).reshape(n, hd) * norm_w.double() * torch.sigmoid(gate), last))
    state = torch.zeros(5, heads, dim, dim, dtype=torch.float32, device=dev)
    state[0] = float("nan")                          # nobody's slot: never read into a result
    slot_of = (3, 1)
    cuts = ([1, 30, 2, 1, 1, 35], [2, 1, 1, 17, 2])
    got = [torch.zeros(n, hd, dtype=torch.float64) for n in lens]
    done = [0, 0]
    for i in range(max(len(c) for c in cuts)):
        who = [s for s in (0, 1) if i < len(cuts[s])]
        counts = [cuts[s][i] for s in who]
        x = torch.cat([projs[s][done[s]:done[s] + c] for s, c in zip(who, counts)])
        cu = [0]
        for c in counts:
            cu.append(cu[-1] + c)
        lead = 0                       # the step's leading one-token sequences: the kernel form of decoded tokens
        while lead < len(counts) and counts[lead] == 1:
            lead += 1
        step = SimpleNamespace(cu_q_lens=torch.tensor(cu, dtype=torch.int32, device=dev),
                               state_slots=torch.tensor([slot_of[s] for s in who], dtype=torch.int32, device=dev),
                               num_seqs=len(who), num_decode=lead)
        y = ops.delta_rule(x.to(dev), w2.to(dt).t().contiguous().to(dev), w0.to(dev), a_bias.to(dev), norm_w.to(dev), state, step,
                           heads, dim, rank, decay_scale, key_eps, eps, dt).cpu().double()
        for j, (s, c) in enumerate(zip(who, counts)):
            got[s][done[s]:done[s] + c] = y[cu[j]:cu[j + 1]]
            done[s] += c
    for s in (0, 1):
        close(got[s], want[s][0], dtype, f"output of sequence {s}", f32=1e-4, bf16=8e-3)
        close(state[slot_of[s]], want[s][1], "float32", f"state of sequence {s}", f32=1e-4)
    assert not torch.isnan(state[1:]).any()


@pytest.mark.parametrize("heads, dim, rank", [(3, 64, 16), (2, 64, 65), (2, 128, 5)])
@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("kind", ["bfloat16", "float32", "split"])
def test_the_delta_rule_of_portions(heads, dim, rank, fast, kind, monkeypatch):
    """Portions of many lengths beside decoded tokens, from states that are not zero, against 64 bits, in the portions'
    form for all sequences too; a sequence's bits do not depend on the others'."""
    from deterministic_inference_b200.kernels import ops
    g, dev, hd = torch.Generator().manual_seed(dim + rank), "cuda", heads * dim
    lens = (1, 1, 2, 47, 48, 49, 111, 112, 113, 129, 160, 150)   # the last one on the padding's slot
    slots = (7, 1, 2, 3, 4, 5, 6, 8, 9, 10, 11, 0)
    w2 = pg.as_stored_bf16(torch.randn(hd, rank, generator=g))
    w0, a_bias = torch.randn(hd, generator=g) + (6.0 if fast else -3.0), torch.randn(hd, generator=g)
    norm_w = 1.0 + 0.1 * torch.randn(hd, generator=g)
    projs = [pg.as_stored_bf16(torch.randn(n, 5 * hd + rank, generator=g)) for n in lens]
    if fast:                                                     # decays at their fastest, e^(-0.6) a token
        for p in projs:
            p[:, 5 * hd:] = 0
    first = torch.randn(12, heads, dim, dim, generator=g)
    first[0] = float("nan")                                      # nobody's slot

    def run(who):
        state = first.to(dev)
        x = torch.cat([projs[i] for i in who]).to(dev)
        if kind == "bfloat16":
            x = x.bfloat16()
        if kind == "split":                                      # two parts whose sum is exact
            x = ops.SplitSum(torch.stack([0.5 * x, 0.5 * x]), torch.float32)
        cu = [0]
        for i in who:
            cu.append(cu[-1] + lens[i])
        step = SimpleNamespace(cu_q_lens=torch.tensor(cu, dtype=torch.int32, device=dev), num_seqs=len(who),
                               state_slots=torch.tensor([slots[i] for i in who], dtype=torch.int32, device=dev),
                               num_decode=sum(lens[i] == 1 for i in who))
        y = ops.delta_rule(x, w2.t().contiguous().to(dev), w0.to(dev), a_bias.to(dev), norm_w.to(dev), state, step, heads,
                           dim, rank, math.exp(-0.5), 1e-6, 2e-5, torch.float32)
        return [y[cu[j]:cu[j + 1]].cpu() for j in range(len(who))], state.cpu()

    everyone = list(range(len(lens)))
    got, state = run(everyone)
    monkeypatch.setattr(ops, "DELTA_FORM", "1")
    by_token, state_by_token = run(everyone)
    monkeypatch.setattr(ops, "DELTA_FORM", "auto")
    # what one order of the float32 sums differs from another by: a token's three sums of dim terms, over the tokens
    # that a state still feels, as sums of squares grow; the root mean square divides both alike
    bound = lambda n: 16 * 2.0 ** -24 * math.sqrt(dim + n)
    for i, n in enumerate(lens):
        p, shape = projs[i].double(), (n, heads, dim)
        r, k, v, gate = (p[:, j * hd:(j + 1) * hd] for j in range(4))
        rate = torch.sigmoid(p[:, 4 * hd:5 * hd] + a_bias.double()).view(shape)
        decay = pg.decay_of(p[:, 5 * hd:], torch.eye(rank, dtype=torch.float64), w2.double(), w0.double()).view(shape)
        start = first[slots[i]].double() if slots[i] else torch.zeros(heads, dim, dim, dtype=torch.float64)
        r, k, v = r.reshape(shape), k.reshape(shape), v.reshape(shape)
        unit, o, s = k / torch.sqrt((k ** 2).sum(-1, keepdim=True) + 1e-6), [], start
        for t in range(n):
            read = torch.einsum("hd,hde->he", unit[t], s)
            s = decay[t][..., None] * s - (rate[t] * unit[t])[..., None] * read[:, None] + k[t][..., None] * v[t][:, None]
            o.append(torch.einsum("hd,hde->he", r[t], s))
        want = pg.unit_rms(torch.stack(o), 2e-5).reshape(n, hd) * norm_w.double() * torch.sigmoid(gate)
        scale = float(want.abs().max())
        assert float((got[i].double() - want).abs().max()) <= bound(n) * scale, (i, n)
        assert float((by_token[i].double() - want).abs().max()) <= bound(n) * scale, (i, n)
        if slots[i]:
            for st in (state, state_by_token):
                assert float((st[slots[i]].double() - s).abs().max()) <= bound(n) * float(s.abs().max()), (i, n)
    assert torch.isnan(state[0]).all()
    for i in (6, 7, 10):
        assert torch.equal(run([i])[0][0], got[i]), i


@pytest.mark.parametrize("heads, dim, rank", [(3, 64, 16), (2, 128, 5), (1, 200, 2)])
@pytest.mark.parametrize("kind", ["bfloat16", "float32", "split"])
def test_the_delta_rule_does_not_see_where_a_prompt_is_cut(heads, dim, rank, kind):
    """A prompt in one portion and in portions of every kind (two tokens, odd ones, multiples of 16): equal bits of every
    token's output and of the state.  The scheduler cuts a prompt to what other requests leave of a step's tokens."""
    from deterministic_inference_b200.kernels import ops
    g, dev, hd, n = torch.Generator().manual_seed(dim + rank), "cuda", heads * dim, 420
    w2 = pg.as_stored_bf16(torch.randn(rank, hd, generator=g)).to(dev)
    w0, a_bias, norm_w = ((torch.randn(hd, generator=g) + x).to(dev) for x in (-3.0, 0.0, 1.0))
    proj = pg.as_stored_bf16(torch.randn(n, 5 * hd + rank, generator=g)).to(dev)
    first = torch.randn(2, heads, dim, dim, generator=g).to(dev)

    def run(cuts):
        state, out = first.clone(), []
        for a, b in zip(cuts, cuts[1:]):
            x = proj[a:b].bfloat16() if kind == "bfloat16" else proj[a:b].contiguous()
            if kind == "split":
                x = ops.SplitSum(torch.stack([0.5 * x, 0.5 * x]), torch.float32)
            step = SimpleNamespace(cu_q_lens=torch.tensor([0, b - a], dtype=torch.int32, device=dev), num_seqs=1,
                                   state_slots=torch.tensor([1], dtype=torch.int32, device=dev), num_decode=0, q_lens=[b - a])
            out.append(ops.delta_rule(x, w2, w0, a_bias, norm_w, state, step, heads, dim, rank, math.exp(-0.5), 1e-6, 2e-5,
                                      torch.float32))
        return torch.cat(out), state

    whole, state = run([0, n])
    for cuts in ([0, 256, n], [0, 100, 300, n], [0, 333, n], [0, 2, 5, 117, n], [0, 129, 131, 250, n]):
        y, s = run(cuts)
        assert torch.equal(y, whole) and torch.equal(s, state), cuts


def test_bits_of_a_token_do_not_depend_on_its_portion_without_the_library(tmp_path):
    """Under ``library_products=False`` the logits of a request in portions of 512 and of 100 are equal bit for bit."""
    from deterministic_inference_b200 import EngineConfig
    from deterministic_inference_b200.engine.batch import SequenceInput
    from deterministic_inference_b200.engine.runner import ModelRunner
    from deterministic_inference_b200.config import GamilornConfig
    from deterministic_inference_b200.kernels import gemm_bf16
    from deterministic_inference_b200.weights import write_random_model
    layer = {"type": "parallel", "mlp": {"kind": "dense", "ff": 256},
             "mixer": {"left": {"heads": 2, "kv_heads": 1, "dim": 64, "vdim": 64, "scale": 0.125,
                                "mask": {"size": 150, "keep_first": 3}},
                       "left_scale": 1.0, "right": {"heads": 4, "dim": 64, "decay_rank": 16}, "right_scale": 1.0}}
    write_random_model(GamilornConfig.from_dict({"architecture": "Gamilorn", "vocab": 160, "width": 256, "max_positions": 1024,
                                                 "norm": {"eps": 1e-5}, "logit_softcap": 30.0,
                                                 "layers": [layer, layer]}), 57, tmp_path)
    tokens = torch.randint(0, 160, (612,), generator=torch.Generator().manual_seed(58)).tolist()
    rows = {}
    try:
        for portion in (512, 100):
            r = ModelRunner(EngineConfig(model_path=str(tmp_path), dtype="bfloat16", kv_pool_tokens=2048, page_size=16,
                                         max_reqs=4, max_seq_len=1024, cuda_graphs=False, library_products=False))
            slot, got = r.cache.allocate_slot(), []
            for c in range(0, len(tokens), portion):
                n = min(portion, len(tokens) - c)
                got.append(r.step([SequenceInput(slot, tokens[c:c + n], c, list(range(n)))])[0].clone())
            rows[portion] = torch.cat(got)
    finally:
        gemm_bf16.set_library_products(True)
    assert torch.equal(rows[512], rows[100])


def prepared(proj, heads, dim, rank, w2_t, w0, a_bias):
    """The delta rule's vectors [tokens, heads, 6, dim] by the kernel; ``proj`` float32 or bfloat16 [tokens, width], or
    float32 split sums [splits, tokens, width]."""
    from ctypes import c_float, c_int, c_longlong

    from deterministic_inference_b200.kernels import ops
    splits, n = (1, proj.shape[0]) if proj.dim() == 2 else proj.shape[:2]
    out = torch.full((n, heads, 6, dim), float("nan"), device=proj.device)
    st = ops._lib("delta_rule").dib_delta_prepare(
        ops._ptr(proj), c_int(1 if proj.dtype == torch.bfloat16 else 0), c_int(splits), c_longlong(proj.stride(0) if splits > 1 else 0),
        ops._ptr(w2_t), c_int(1 if w2_t.dtype == torch.bfloat16 else 0), ops._ptr(w0), ops._ptr(a_bias), ops._ptr(out),
        c_int(n), c_int(heads), c_int(dim), c_int(rank), c_float(math.exp(-0.5)), c_float(1e-6), ops._stream())
    assert st == 0, st
    return out


def prepared_in_64_bits(proj, heads, dim, rank, w2_t, w0, a_bias):
    p, hd = proj.double(), heads * dim
    r, k, v = (p[:, i * hd:(i + 1) * hd].view(-1, heads, dim) for i in range(3))
    rate = torch.sigmoid(p[:, 4 * hd:5 * hd] + a_bias.double()).view(-1, heads, dim)
    w = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(p[:, 5 * hd:]) @ w2_t.double() + w0.double()))
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    return torch.stack([w.view(-1, heads, dim), rate * u, u, k, r, v], dim=2)


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("dim", [256, 257, 1000, 1024])
def test_the_delta_rules_vectors_of_wide_heads(dim, dtype):
    """Every head size the call accepts: a block of up to 1,024 threads has the registers it needs."""
    g = torch.Generator(device="cuda").manual_seed(dim)
    rank, heads, n = 12, 2, 11
    proj = torch.randn(n, 5 * heads * dim + rank, generator=g, device="cuda").to(DTYPES[dtype])
    w2_t = torch.randn(rank, heads * dim, generator=g, device="cuda").to(DTYPES[dtype])
    w0, a_bias = torch.randn(heads * dim, generator=g, device="cuda") - 2, torch.randn(heads * dim, generator=g, device="cuda")
    got = prepared(proj, heads, dim, rank, w2_t, w0, a_bias)
    want = prepared_in_64_bits(proj, heads, dim, rank, w2_t, w0, a_bias)
    # a chain of `rank` terms of size |w2| <= 5 into the decay; a few roundings elsewhere
    assert float((got.double() - want).abs().max()) <= (5 * rank + 32) * 2.0 ** -24 * float(want.abs().max())


@pytest.mark.parametrize("heads, dim, rank", [(3, 64, 64), (2, 40, 513), (1, 256, 0), (2, 20, 7)])
def test_the_delta_rules_vectors_in_every_form(heads, dim, rank):
    """One, two or four tokens a block, by the step's tokens, stored projections of both types and split sums: a token's
    vectors are those of the token alone, at the edges of the blocks and of the hidden vector's runs; split sums give
    what their sum in split order gives, and all are 64 bits' up to rounding."""
    g = torch.Generator(device="cuda").manual_seed(dim + rank)
    hd, width, n = heads * dim, 5 * heads * dim + rank, 387
    parts = torch.randn(3, n, width, generator=g, device="cuda")
    total = (parts[0] + parts[1]) + parts[2]
    w2_t = torch.randn(rank, hd, generator=g, device="cuda").bfloat16()
    w0, a_bias = torch.randn(hd, generator=g, device="cuda") - 2, torch.randn(hd, generator=g, device="cuda")
    run = lambda x: prepared(x, heads, dim, rank, w2_t, w0, a_bias)
    whole = run(total)
    want = prepared_in_64_bits(total, heads, dim, rank, w2_t, w0, a_bias)
    # a chain of `rank` terms of size |w2| <= 5 into the decay; a few roundings elsewhere
    assert float((whole.double() - want).abs().max()) <= (5 * rank + 32) * 2.0 ** -24 * float(want.abs().max())
    assert torch.equal(run(parts), whole)
    for m in (1, 2, 3, 8, 65, 383, 384, 385, 386):
        assert torch.equal(run(total[:m]), whole[:m]), m
        assert torch.equal(run(parts[:, :m].contiguous()), whole[:m]), m
    stored = total.bfloat16()
    rounded = run(stored)
    assert torch.equal(rounded, run(stored.float()))
    for m in (1, 383):
        assert torch.equal(run(stored[:m]), rounded[:m]), m


@pytest.mark.parametrize("heads, dim", [(16, 64), (3, 20), (2, 128), (1, 100), (2, 200)])
@pytest.mark.parametrize("splits", [2, 4, 5, 8, 11])
def test_the_delta_rules_output_from_split_sums(heads, dim, splits):
    """The gate as split sums gives the bits of their sum in split order, for any number of splits."""
    from ctypes import c_float, c_int, c_longlong

    from deterministic_inference_b200.kernels import ops
    g = torch.Generator(device="cuda").manual_seed(dim + splits)
    n, rank, hd = 5, 3, heads * dim
    parts = torch.randn(splits, n, 5 * hd + rank, generator=g, device="cuda")
    total = parts[0].clone()
    for x in parts[1:]:
        total += x
    o, norm_w = torch.randn(n, hd, generator=g, device="cuda"), torch.rand(hd, generator=g, device="cuda")

    def run(proj, k):
        out = torch.full((n, hd), float("nan"), device="cuda")
        st = ops._lib("delta_rule").dib_delta_output(
            ops._ptr(o), ops._ptr(proj), c_int(0), c_int(k), c_longlong(total.numel()), ops._ptr(norm_w), ops._ptr(out),
            c_int(0), c_int(n), c_int(heads), c_int(dim), c_int(rank), c_float(1e-6), ops._stream())
        assert st == 0, st
        return out

    got = run(total, 1)
    assert torch.equal(run(parts, splits), got)
    x = o.double().view(n, heads, dim)
    want = (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)).reshape(n, hd) * norm_w.double() * \
        torch.sigmoid(total[:, 3 * hd:4 * hd].double())
    # a norm over up to 200 elements and a few roundings
    assert float((got.double() - want).abs().max()) <= (dim / 2 + 16) * 2.0 ** -24 * float(want.abs().max())


# ---- whole models through the trace runner -----------------------------------------------------------

CASES = {
    "g1": ([1, 2, 17, 48, 131, 260], 31),
    "g2": ([5, 33, 64, 200], 32),
    "g3": ([3, 22, 57, 130, 333], 33),
    "g4": ([1, 9, 40, 150], 34),
}


def row_error(got, want):
    d = got.double() - want.double()
    d = d - d.mean()
    return float(d.pow(2).mean().sqrt())


@pytest.fixture(scope="module")
def plain_logits(model_dirs):
    out = {}
    for name, (lens, seed) in CASES.items():
        cfg, w = pg.read_model_dir(model_dirs[name])
        reqs = gu.requests(cfg["vocab"], lens, seed)
        exact = [pg.forward(cfg, w, r) for r in reqs]
        stored = [pg.forward(cfg, w, r, store_bf16=True) for r in reqs]
        out[name] = (cfg, reqs, exact, stored)
    return out


@pytest.mark.parametrize("dtype", list(DTYPES))
@pytest.mark.parametrize("name", list(CASES))
def test_replay_all_cuttings(name, dtype, model_dirs, plain_logits, tmp_path):
    cfg, reqs, exact, stored = plain_logits[name]
    trace = ru.Trace()
    ru.mixed(trace, reqs)                             # sizes the pool; four live requests at most
    ru.whole(trace, reqs)
    ru.last_one_by_one(trace, reqs, tail=150)         # decoding over more tokens than any window
    ru.portions(trace, reqs)
    out = ru.run_trace(model_dirs[name], dtype, trace, tmp_path / "out", page_size=gu.CONFIGS[name]["page_size"])
    got = ru.read_rows(out, trace, cfg["vocab"])
    for kind in "mwtp":
        for i, r in enumerate(reqs):
            assert all((f"{kind}{i}", p) in got for p in range(len(r))), (kind, i)
    worst = 0.0
    for (key, pos), row in got.items():
        i = int(key[1:])
        scale = float(exact[i].std())
        err = row_error(row, exact[i][pos])
        if dtype == "float32":
            bound = 1e-4 * scale
        else:
            # what bfloat16 storage alone does to this request's logits, three times over
            yard = max(row_error(a, b) for a, b in zip(stored[i], exact[i]))
            bound = max(3.0 * yard, 2e-2 * scale)
        assert err <= bound, f"{name}/{dtype}: request {key} position {pos}: {err:.4g} exceeds {bound:.4g}"
        worst = max(worst, err / scale)
    print(f"{name}/{dtype}: worst difference {worst:.3e} of the logits' spread")


@pytest.mark.parametrize("dtype", list(DTYPES))
def test_greedy_generation_through_the_entry_point(dtype, model_dirs):
    from deterministic_inference_b200 import Engine, EngineConfig, SamplingParams
    d = model_dirs["g3"]
    cfg, w = pg.read_model_dir(d)
    prompts = gu.requests(cfg["vocab"], [3, 40, 9, 77, 15], 9)
    new = 40
    eng = Engine(EngineConfig(model_path=str(d), dtype=dtype, kv_pool_tokens=384, page_size=8, max_reqs=3,
                              max_seq_len=160, max_prefill_tokens=48))
    outs = eng.generate(prompts, SamplingParams(max_new_tokens=new, ignore_eos=True))
    eng.cache.check_invariants()
    for p, o in zip(prompts, outs):
        assert len(o.token_ids) == new
        ids = list(p)
        for t in o.token_ids:
            logits = pg.forward(cfg, w, ids)[-1]
            best = int(torch.argmax(logits))
            if t != best:
                # another token only where rounding can flip the choice; from there on the
                # engine's own continuation is followed
                gap = float(logits[best] - logits[t])
                assert dtype == "bfloat16" and gap < 0.25, f"token {t} instead of {best}, logits {gap:.3g} apart"
            ids.append(t)
