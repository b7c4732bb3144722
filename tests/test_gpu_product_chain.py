"""The resident kernel of consecutive products (csrc/product_chain.cu) and the host side that lets them wait for one another."""
import contextlib

import numpy as np
import pytest
import torch

import harness as H
from zekivik_configs import ALL as ZEKIVIK

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from lastengine_b200.ops import kernels
    return kernels


# ---- code from elsewhere inside a step ---------------------------------------------------------------------
def torch_gate(block_gate, kept):
    """The sigmoid gate in plain torch, with a copy of what it read."""
    from lastengine_b200.parts.gate import SigmoidGate

    class TorchGate(SigmoidGate):
        def add_gated(self, x, y, h, env, z=None, next_norm=None, h_out=None):
            z = h.float() @ self.w.float().T if z is None else z.float()
            kept.append(y.clone())
            x += y * torch.sigmoid(z + self.b if self.b is not None else z)
            if h_out is not None:
                next_norm.forward(h_out, x)
    block_gate.__class__ = TorchGate


def wrapped(part, kept):
    """A part's forward as a caller wraps it to look at what goes in and comes out."""
    own = part.forward

    def forward(h, out, *a, **k):
        kept.append(h.clone())
        own(h, out, *a, **k)
        kept.append(out.clone())
    part.forward = forward


@pytest.mark.parametrize("rows", [17, 64])
@pytest.mark.parametrize("what", ["gate", "wrapped"])
def test_code_from_elsewhere_reads_finished_products(what, rows, tmp_path, monkeypatch):
    """A gate in plain torch, and a feed-forward wrapped to keep copies of its operands, put into a built model: in steps whose
    products wait for one another they read what those products give.  Against the same model with every product launched
    at its call; the step before it had other tokens, so that a buffer read too early holds other numbers.  Whole rows agree to
    the rounding of a bfloat16 model (K is cut differently in a chain)."""
    from lastengine_b200 import Engine
    from lastengine_b200.weights import write_model_dir
    k = K()
    name = next(n for n, c in ZEKIVIK.items() if sum(lay["mlp"] is not None for lay in c["layers"]) > 1)
    cfg = ZEKIVIK[name]
    d = write_model_dir(cfg, str(tmp_path), seed=3, norm_init="random")
    rng = np.random.default_rng(rows)
    prompts = [rng.integers(0, cfg["vocab"], size=rows).tolist() for _ in range(2)]

    def run():
        eng = Engine.from_pretrained(d, dtype="bfloat16", max_tokens=512)
        H.run_whole(eng, prompts[0])       # (a first step: matrices that a gate gives to a mixer have moved)
        kept: list = []
        for block in eng.model.blocks:
            if what == "wrapped":
                for part in (block.mixer, block.ffn):
                    if part is not None:
                        wrapped(part, kept)
            else:
                for gate in (block.mixer_gate, block.ffn_gate):
                    if gate is not None:
                        torch_gate(gate, kept)
        H.run_whole(eng, prompts[0])
        kept.clear()
        logits = H.run_whole(eng, prompts[1])
        k.check_device_status()
        return logits, [t.float().cpu() for t in kept]
    got = run()
    monkeypatch.setattr(k, "product_chain", lambda *a: contextlib.nullcontext())
    want = run()
    assert len(got[1]) == len(want[1]) >= 2
    for a, b in zip(got[1] + [got[0]], want[1] + [want[0]]):
        e = (a - b).abs().amax(-1) / b.abs().max()
        assert e.median() < H.TOL_BF16 / 3 and torch.quantile(e, 0.9) < 2 * H.TOL_BF16


# ---- the kernel --------------------------------------------------------------------------------------------
def gen(*shape, seed, scale=1.0, dtype=torch.bfloat16):
    g = torch.Generator().manual_seed(seed)
    return (scale * torch.randn(*shape, generator=g)).to(dtype).to(DEV)


def workspace():
    from lastengine_b200.engine.workspace import Workspace
    return Workspace(torch.device(DEV))


@pytest.mark.parametrize("M", [17, 64, 65, 128])
def test_slices_without_k_between_others(M):
    """Products of so few k that some blocks of a cluster have none (up to 192, 257 to 384, 513 to 576), of several tiles a
    cluster, between products of many k: each against 64 bits (up to K bfloat16 terms in float), and the same bits every time."""
    k, ws = K(), workspace()
    inner = (2048, 64, 192, 2048, 320, 576, 128, 2048, 64, 2048)
    outer = (64, 192, 2048, 320, 576, 128, 2048, 64, 2048, 12672)
    W = [gen(n, kk, seed=i, scale=kk ** -0.5) for i, (n, kk) in enumerate(zip(outer, inner))]
    h = gen(M, inner[0], seed=50)
    first = None
    for _ in range(20):
        outs, x = [], h
        with k.product_chain(ws, M, torch.bfloat16):
            for i, w in enumerate(W):
                outs.append(torch.empty(M, w.shape[0], device=DEV, dtype=torch.float32 if i == len(W) - 1 else torch.bfloat16))
                k.linear(outs[-1], x, w)
                x = outs[-1]
        first = first or outs
        assert all(torch.equal(a, b) for a, b in zip(first, outs))
    k.check_device_status()
    for x, w, y in zip([h, *first], W, first):
        want = x.double() @ w.double().T
        tol = 2 ** -8 + 2e-5 if y.dtype == torch.bfloat16 else 2e-5
        assert float((y.double() - want).abs().max() / want.abs().max()) < tol


@pytest.mark.parametrize("N,kk", [(64, 64), (328, 4224), (512, 8192), (768, 3072), (1000, 5000), (2048, 2048), (2048, 5632), (2048, 7168),
                                  (3072, 2048), (2560, 9728)])
@pytest.mark.parametrize("M", [17, 64, 128])
def test_a_chained_product_is_as_near_to_64_bits_as_one_alone(M, N, kk):
    """K is cut otherwise in a chain, but no accumulator takes more of it than a slice of the product alone: one to eight of them in
    a block's slice, ends between the two k-blocks of a stage, and (512 x 8,192 at 128 rows) more than a chain takes.  The same operands on
    both sides; 1.05 for the draw of the roundings (measured: 0.22 to 1.00; with one accumulator a slice 1.4 to 8.4)."""
    k, ws = K(), workspace()
    W, h = gen(N, kk, seed=kk, scale=kk ** -0.5), gen(M, kk, seed=M)
    want = h.double() @ W.double().T
    off = {}
    for chained in (True, False):
        outs = [torch.empty(M, N, device=DEV) for _ in range(6)]
        before = k.launch_count()
        with k.product_chain(ws, M, torch.bfloat16) if chained else contextlib.nullcontext():
            for y in outs:
                k.linear(y, h, W)
        assert (k.launch_count() - before == 1) == (chained and not (kk == 8192 and M == 128))
        assert all(torch.equal(outs[0], y) for y in outs)
        off[chained] = float((outs[0].double() - want).norm() / want.norm())
    k.check_device_status()
    assert off[True] <= 1.05 * off[False]


@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("Lc", [2, 3, 4, 5])
@pytest.mark.parametrize("M,D", [(17, 520), (64, 1024), (97, 776)])
def test_convolutions_in_a_chain(M, D, Lc, bias):
    """The one-token convolution as a chain's epilogue for every number of taps, with and without an additive term: results and states of
    two steps against 64 bits from the projections as bfloat16 (a projection may be rounded to either side: half a step, 2^-9 of the
    largest, in each of the three factors), slots in another order than the rows, a padding row."""
    import types
    k, ws = K(), workspace()
    w_in, w_out = gen(3 * D, D, seed=1, scale=D ** -0.5), gen(D, D, seed=2, scale=D ** -0.5)
    taps, b = gen(D, Lc, seed=3, dtype=torch.float32), gen(D, seed=4, scale=0.1, dtype=torch.float32) if bias else None
    slot = torch.arange(M, dtype=torch.int32).flip(0)
    slot[M // 2] = -1
    batch = types.SimpleNamespace(max_qlen=1, n_seqs=M, row_seq=torch.arange(M, dtype=torch.int32, device=DEV), seq_slot=slot.to(DEV))
    state = gen(M, D, Lc - 1, seed=5, dtype=torch.float32)
    want_state, on = state.double().cpu(), slot >= 0
    for step in range(2):
        h = gen(M, D, seed=6 + step)
        y, x, before = torch.empty(M, D, dtype=torch.bfloat16, device=DEV), [torch.zeros(M, D, device=DEV) for _ in range(5)], k.launch_count()
        with k.product_chain(ws, M, torch.bfloat16):
            assert k.shortconv_decode_fused(y, h, w_in, taps, b, state, batch, Lc)
            for t in x:
                k.linear(t, y, w_out, k.ACCUMULATE)
        assert k.launch_count() - before == 1
        pb, pc, pu = (h.double().cpu() @ w_in.double().cpu().T).to(torch.bfloat16).double().chunk(3, -1)
        bu, old = pb * pu, want_state[slot.clamp(min=0).long()]
        row = torch.cat([old, bu[:, :, None]], -1)
        conv = (row * taps.double().cpu()).sum(-1) + (b.double().cpu() if bias else 0.0)
        want = torch.where(on[:, None], pc * conv, torch.zeros(()).double())
        assert float((y.double().cpu() - want).abs().max() / want.abs().max()) < 4 * 2 ** -8
        want_state = want_state.clone()
        want_state[slot[on].long()] = row[on][:, :, 1:]
        assert float((state.double().cpu() - want_state).abs().max() / want_state.abs().max()) < 2 * 2 ** -8
        state.copy_(want_state)
        assert float((x[-1].double() - y.double() @ w_out.double().T).abs().max() / x[-1].abs().max()) < 2e-5
    k.check_device_status()


def chain_of(k, ws, h, W, gate, norm):
    """Six products with both halves of a split norm; the results of every one."""
    M, D = h.shape
    x = torch.zeros(M, D, device=DEV)
    sp = k.SplitNorm(torch.empty(M, D, dtype=torch.bfloat16, device=DEV), torch.empty(M, -(-D // 16), device=DEV), norm, 1e-5)
    a = torch.empty(M, gate.shape[0] // 2, dtype=torch.bfloat16, device=DEV)
    z = [torch.empty(M, D, device=DEV) for _ in range(4)]
    with k.product_chain(ws, M, torch.bfloat16):
        k.linear(x, h, W, k.ACCUMULATE, emit=sp)
        k.linear(a, sp.values, gate, k.SWIGLU, scale=sp)
        for t in z:
            k.linear(t, sp.values, W, scale=sp)
    return [x, sp.values, sp.ssq, a, *z]


@pytest.mark.parametrize("D,F", [(520, 1040), (2048, 2816)])
def test_a_row_of_a_chain_does_not_depend_on_the_others(D, F):
    """The same bits at every padding of the rows, alone with others' rows beside them."""
    k, ws = K(), workspace()
    W, gate, norm = gen(D, D, seed=1, scale=D ** -0.5), gen(2 * F, D, seed=2, scale=D ** -0.5), 1 + gen(D, seed=3, scale=0.1, dtype=torch.float32)
    h = gen(128, D, seed=4)
    want = chain_of(k, ws, h, W, gate, norm)
    for M in (17, 32, 33, 64, 65, 96, 97):
        for lo in (0, 128 - M):
            for got, all_ in zip(chain_of(k, ws, h[lo:lo + M].contiguous(), W, gate, norm), want):
                assert torch.equal(got, all_[lo:lo + M])
    k.check_device_status()


def test_chains_longer_than_the_kernel_takes_and_of_one_product():
    """A chain that is full is launched and the next one begins (40 products); one product that leaves a norm's half is launched alone."""
    k, ws, M, D = K(), workspace(), 40, 264
    W, h = gen(D, D, seed=1, scale=D ** -0.5), gen(M, D, seed=2)
    most = k.lib().leb_chain_max_ops()
    outs, x, before = [torch.empty(M, D, dtype=torch.bfloat16, device=DEV) for _ in range(2 * most + 7)], h, k.launch_count()
    with k.product_chain(ws, M, torch.bfloat16):
        for y in outs:
            k.linear(y, x, W)
            x = y
    assert k.launch_count() - before == 3
    for x, y in zip([h, *outs], outs):
        want = x.double() @ W.double().T
        assert float((y.double() - want).abs().max() / want.abs().max()) < 2 ** -8 + 2e-5
    results = []
    for chained in (True, False):
        s = torch.zeros(M, D, device=DEV)
        sp = k.SplitNorm(torch.empty(M, D, dtype=torch.bfloat16, device=DEV), torch.empty(M, -(-D // 16), device=DEV), torch.ones(D, device=DEV), 1e-5)
        with k.product_chain(ws, M, torch.bfloat16) if chained else contextlib.nullcontext():
            k.linear(s, h, W, k.ACCUMULATE, emit=sp)
        assert sp.filled
        results.append((s, sp.values, sp.ssq))
    assert all(torch.equal(a, b) for a, b in zip(*results))
    k.check_device_status()


def test_a_step_that_raises_launches_nothing_and_the_next_chain_is_whole():
    k, ws, M, D = K(), workspace(), 40, 264
    W, h = gen(D, D, seed=1, scale=D ** -0.5), gen(M, D, seed=2)
    y = [torch.full((M, D), 7.0, device=DEV) for _ in range(5)]
    before = k.launch_count()
    with pytest.raises(ValueError), k.product_chain(ws, M, torch.bfloat16):
        for t in y:
            k.linear(t, h, W)
        raise ValueError
    assert k.launch_count() == before and all(bool((t == 7).all()) for t in y)
    with k.product_chain(ws, M, torch.bfloat16):
        for t in y:
            k.linear(t, h, W)
    want = h.double() @ W.double().T
    assert all(float((t.double() - want).abs().max() / want.abs().max()) < 2e-5 for t in y)
    k.check_device_status()


def test_a_chain_whose_barrier_is_never_passed_gives_up():
    """The grid barrier's count put where no arrival brings it to its target: every block gives its bounded wait up (after about a
    second), the status word says so, the context and the barrier's words are usable, and the next chain is right."""
    k, ws, M, D = K(), workspace(), 40, 264
    W, h = gen(D, D, seed=1, scale=D ** -0.5), gen(M, D, seed=2)
    y = [torch.empty(M, D, device=DEV) for _ in range(5)]

    def run():
        with k.product_chain(ws, M, torch.bfloat16):
            for t in y:
                k.linear(t, h, W)
    k.check_device_status()
    ws.zeroed("chain.sync", 2)[0] = -1000
    run()
    torch.cuda.synchronize()
    with pytest.raises(k.KernelError, match=r"role 4\d"):
        k.check_device_status()
    assert ws.zeroed("chain.sync", 2).tolist() == [0, 0]
    run()
    k.check_device_status()
    want = h.double() @ W.double().T
    assert all(float((t.double() - want).abs().max() / want.abs().max()) < 2e-5 for t in y)
