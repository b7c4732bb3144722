"""Each kernel alone against plain arithmetic, at sizes the tiny models do not use:
widths and vocabularies that are no power of two, head sizes 16/48/80, odd group sizes,
rows that are no multiple of any tile."""
import math

import numpy as np
import pytest
import torch

import harness as H  # noqa: F401  (path setup)
import plain_lfm3 as P

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def K():
    from lastengine_b200.ops import kernels
    return kernels


def builder():
    from lastengine_b200.engine.batch import BatchBuilder
    return BatchBuilder(torch.device(DEV))


def gen(*shape, seed=0, scale=1.0, dtype=torch.float32):
    g = torch.Generator().manual_seed(seed)
    return (scale * torch.randn(*shape, generator=g)).to(dtype)


def err(got, want):
    got, want = got.double().cpu(), want.double().cpu()
    return float((got - want).abs().max() / (want.abs().max() + 1e-30))


# ---- rows ------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embed(dtype):
    table = gen(301, 72, seed=1).to(dtype)
    toks = torch.tensor([0, 300, 17, 17, 5], dtype=torch.int32)
    x = torch.empty(5, 72, device=DEV)
    K().embed(x, table.to(DEV), toks.to(DEV))
    assert torch.equal(x.cpu(), table.float()[toks.long()])


@pytest.mark.parametrize("D", [100, 64, 2048, 5000])
def test_rmsnorm(D):
    x, w = gen(7, D, seed=2, scale=3.0), 1 + 0.1 * gen(D, seed=3)
    want = P.rms_norm(x.double(), w.double(), 1e-3)
    out = torch.empty(7, D, device=DEV)
    K().rmsnorm(out, x.to(DEV), w.to(DEV), 1e-3)
    assert err(out, want) < 1e-6
    ob = torch.empty(7, D, device=DEV, dtype=torch.bfloat16)
    K().rmsnorm(ob, x.to(DEV), w.to(DEV), 1e-3)
    assert err(ob, want) < 5e-3                     # its own order of sums: equal up to one bfloat16 rounding
    rows = torch.tensor([6, 0, 3], dtype=torch.int32, device=DEV)
    o3 = torch.empty(3, D, device=DEV)
    K().rmsnorm(o3, x.to(DEV), w.to(DEV), 1e-3, rows=rows)
    assert torch.equal(o3.cpu(), out.cpu()[[6, 0, 3]])
    res = gen(7, D, seed=4).to(DEV)
    r0 = res.clone()
    K().rmsnorm(res, x.to(DEV), w.to(DEV), 1e-3, add=True)
    assert err(res, r0.cpu().double() + want) < 1e-6


@pytest.mark.parametrize("D", [2052, 4096, 8192])
def test_rmsnorm_of_many_rows_gives_the_bits_of_few(D):
    """Few rows fetch the weights ahead of the wait for the kernel before, many do not (more than fit the SMs at once)."""
    x, w = gen(3001, D, seed=2, dtype=torch.float32).to(DEV), (1 + 0.1 * gen(D, seed=3)).to(DEV)
    many, few = (torch.empty(3001, D, device=DEV, dtype=torch.bfloat16) for _ in range(2))
    K().rmsnorm(many, x, w, 1e-3)
    for r in range(0, 3001, 100):
        K().rmsnorm(few[r:r + 100], x[r:r + 100], w, 1e-3)
    assert torch.equal(many, few)


def test_swiglu():
    gu = gen(9, 2 * 37, seed=5, scale=2.0)
    want = P.silu(gu[:, :37].double()) * gu[:, 37:].double()
    out = torch.empty(9, 37, device=DEV)
    K().swiglu(out, gu.to(DEV))
    assert err(out, want) < 1e-6
    ob = torch.empty(9, 37, device=DEV, dtype=torch.bfloat16)
    K().swiglu(ob, gu.to(DEV))
    assert err(ob, want) < 5e-3


# ---- matrix products ---------------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K_", [(1, 50, 70), (37, 129, 33), (64, 64, 16), (130, 70, 200)])
def test_linear_f32(M, N, K_):
    x, w = gen(M, K_, seed=6), gen(N, K_, seed=7)
    want = x.double() @ w.double().T
    out = torch.empty(M, N, device=DEV)
    K().linear(out, x.to(DEV), w.to(DEV))
    assert err(out, want) < 2e-6
    base = gen(M, N, seed=8).to(DEV)
    b0 = base.clone()
    K().linear(base, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    assert err(base, b0.cpu().double() + want) < 2e-6
    # a row's result does not depend on the other rows of the launch
    one = torch.empty(1, N, device=DEV)
    K().linear(one, x[M - 1:].to(DEV), w.to(DEV))
    assert torch.equal(one.cpu()[0], out.cpu()[M - 1])


@pytest.mark.parametrize("M", [1, 2, 4, 8, 9, 16, 17, 32, 33, 64, 65, 129, 300])
@pytest.mark.parametrize("N,K_", [(17, 4), (50, 124), (2400, 128), (36, 132), (130, 2052), (4111, 260), (33, 4100), (40, 301)])
def test_linear_f32_sums(M, N, K_):
    """The 32-bit product around the borders of its kernels' tiles (every one of them runs in the test below): part tiles, part chunks of k, more chunks than a round holds, rows with a stride, and the same bits
    whatever the row count.  A chunk of up to 128 products and a sum over K/128 chunks: each rounding is at most 2^-24
    of a partial sum, so 2^-24 * (128 + K/128) of sum |x w| bounds every element."""
    x, w = gen(M, K_ + 12, seed=6)[:, :K_], gen(N, K_, seed=7)
    want = x.double() @ w.double().T
    bound = 2.0 ** -24 * (min(K_, 128) + K_ / 128 + 2) * (x.double().abs() @ w.double().abs().T)
    xd, wd = gen(M, K_ + 12, seed=6).to(DEV)[:, :K_], w.to(DEV)
    out = torch.full((M, N), float("nan"), device=DEV)
    K().linear(out, xd, wd)
    assert bool(((out.cpu().double() - want).abs() <= bound).all())
    base = gen(M, N, seed=8).to(DEV)
    b0 = base.clone()
    K().linear(base, xd, wd, K().ACCUMULATE)
    assert torch.equal(base, b0 + out)
    one = torch.empty(1, N, device=DEV)
    K().linear(one, xd[M - 1:], wd)
    assert torch.equal(one[0], out[M - 1])
    # rows grouped by expert: each group against its own weights, an empty group among them
    offs = torch.tensor([0, M // 3, M // 3, M], dtype=torch.int32, device=DEV)
    w3 = torch.stack([wd, wd * 2, wd * 0.5])
    grouped = torch.full((M, N), float("nan"), device=DEV)
    K().linear(grouped, xd, w3, group_offsets=offs)
    assert torch.equal(grouped[:M // 3], out[:M // 3]) and torch.equal(grouped[M // 3:], out[M // 3:] * 0.5)


# (rows, columns, inner size, kernel as leb_gemm_f32_choice numbers them: 0 tiles of 128 x 128, 1 of 64 x 64, 2 of 32 x 32, 3 of 64 x 16,
# 4 of 32 x 16, 5 blocks of 64 x 64 by the SM, 6 the stream), the same on GPUs of 144 to 152 SMs; inner sizes that are no
# multiple of four have no whole 16-byte vectors
F32_KERNELS = [(69, 10244, 252, 0), (145, 6821, 252, 0), (65, 11264, 516, 0), (288, 650, 416, 1), (1031, 300, 1028, 1),
               (133, 767, 268, 2), (300, 300, 1028, 2), (2557, 36, 200, 3), (1757, 65, 300, 3), (33, 17, 132, 4), (138, 3, 204, 4),
               (300, 2048, 128, 5), (523, 1500, 4, 5), (67, 65, 100, 5), (9, 1, 1084, 6), (8, 300, 60, 6), (16, 17, 2388, 6),
               (340, 5111, 118, 0), (606, 3455, 510, 0), (9, 5311, 443, 1), (627, 305, 477, 1), (170, 643, 329, 2), (2502, 35, 283, 3),
               (27, 5, 737, 4), (300, 771, 301, 5), (964, 2, 5, 5)]
F32_GROUPED = [(1000, 512, 512, 1), (300, 768, 516, 2), (40, 512, 1028, 4), (64, 64, 64, 5), (300, 1023, 61, 5)]


@pytest.mark.parametrize("M,N,K_,kind", F32_KERNELS)
def test_linear_f32_every_kernel(M, N, K_, kind):
    """Each kernel of the 32-bit product, where the choice takes it, with and without whole 16-byte vectors: against 64 bits
    (the bound of the test above) and the bits of its rows alone, which another kernel computes."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert K().lib().leb_gemm_f32_choice(M, N, K_, 0, int(K_ % 4 == 0), sms) == kind
    xd, wd = gen(M, K_, seed=6).to(DEV), gen(N, K_, seed=7).to(DEV)
    out = torch.full((M, N), float("nan"), device=DEV)
    K().linear(out, xd, wd)
    want = xd.double() @ wd.double().T
    bound = 2.0 ** -24 * (min(K_, 128) + K_ / 128 + 2) * (xd.double().abs() @ wd.double().abs().T)
    assert bool(((out.double() - want).abs() <= bound).all())
    for m in (0, M // 2, M - 1):
        one = torch.empty(1, N, device=DEV)
        K().linear(one, xd[m:m + 1], wd)
        assert torch.equal(one[0], out[m])
    base = gen(M, N, seed=8).to(DEV)
    b0 = base.clone()
    K().linear(base, xd, wd, K().ACCUMULATE)
    assert torch.equal(base, b0 + out)


@pytest.mark.parametrize("M,N,K_,kind", F32_GROUPED)
def test_linear_f32_every_grouped_kernel(M, N, K_, kind):
    """... and the kernels that take products grouped by expert: unequal groups, an empty one and a single row among
    them, the bits of the ungrouped product."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert K().lib().leb_gemm_f32_choice(M, N, K_, 4, int(K_ % 4 == 0), sms) == kind
    xd, wd = gen(M, K_, seed=6).to(DEV), gen(N, K_, seed=7).to(DEV)
    plain = torch.empty(M, N, device=DEV)
    K().linear(plain, xd, wd)
    at = [0, M // 3, M // 3, M - 1, M]
    out = torch.full((M, N), float("nan"), device=DEV)
    K().linear(out, xd, torch.stack([wd, wd * 4, wd * 2, wd * 0.5]), group_offsets=torch.tensor(at, dtype=torch.int32, device=DEV))
    for e, f in enumerate((1, 4, 2, 0.5)):
        assert torch.equal(out[at[e]:at[e + 1]], plain[at[e]:at[e + 1]] * f)


def test_one_f32_group_is_its_rows_alone():
    """A single group may begin and end inside the rows: up to 8 of them, where the ungrouped product streams its weights."""
    x, w = gen(6, 64, seed=6).to(DEV), gen(40, 64, seed=7).to(DEV)
    out = torch.full((6, 40), -7.0, device=DEV)
    K().linear(out, x, w[None], group_offsets=torch.tensor([2, 5], dtype=torch.int32, device=DEV))
    whole = torch.empty(6, 40, device=DEV)
    K().linear(whole, x, w)
    assert torch.equal(out[2:5], whole[2:5]) and bool((out[:2] == -7).all()) and bool((out[5:] == -7).all())


@pytest.mark.parametrize("M", [1, 5, 8, 9, 33, 64, 65, 200])
@pytest.mark.parametrize("N,K_", [(48, 72), (100, 200), (17, 40)])
def test_linear_bf16_small(M, N, K_):
    x, w = gen(M, K_, seed=9, dtype=torch.bfloat16), gen(N, K_, seed=10, dtype=torch.bfloat16)
    want = x.double() @ w.double().T
    out = torch.empty(M, N, device=DEV)
    K().linear(out, x.to(DEV), w.to(DEV), streaming=True)
    assert err(out, want) < 1e-5
    ob = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    K().linear(ob, x.to(DEV), w.to(DEV), streaming=True)
    assert err(ob, want) < 5e-3
    base = gen(M, N, seed=11).to(DEV)
    b0 = base.clone()
    K().linear(base, x.to(DEV), w.to(DEV), K().ACCUMULATE, streaming=True)
    assert err(base, b0.cpu().double() + want) < 1e-5
    one = torch.empty(1, N, device=DEV)
    K().linear(one, x[M - 1:].to(DEV), w.to(DEV), streaming=True)
    assert torch.equal(one.cpu()[0], out.cpu()[M - 1])


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("N,K_", [(48, 72), (100, 200), (17, 40), (2048, 2048), (6144, 136), (352, 5632), (9600, 64)])
def test_linear_bf16_stream(M, N, K_):
    """The decode product (weights through rings of asynchronous copies): widths that leave part
    of a tile, K that leaves part of a chunk or gives some warps nothing, more tiles than blocks."""
    x, w = gen(M, K_, seed=9, dtype=torch.bfloat16), gen(N, K_, seed=10, scale=0.05, dtype=torch.bfloat16)
    want = x.double() @ w.double().T
    out = torch.full((M, N), float("nan"), device=DEV)
    K().linear(out, x.to(DEV), w.to(DEV))
    assert err(out, want) < 1e-5
    ob = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    K().linear(ob, x.to(DEV), w.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(M, N, seed=11).to(DEV)
    b0 = base.clone()
    K().linear(base, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    assert err(base, b0.cpu().double() + want) < 1e-5
    one = torch.empty(1, N, device=DEV)
    K().linear(one, x[M - 1:].to(DEV), w.to(DEV))
    assert torch.equal(one.cpu()[0], out.cpu()[M - 1])      # a row does not depend on the other rows
    if N % 32 == 0:
        from lastengine_b200.parts.ffn import fuse_gate_up
        F = N // 2
        w13 = fuse_gate_up(w[:F], w[F:], True).to(DEV)
        sw = P.silu(want[:, :F]) * want[:, F:]
        o2 = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
        K().linear(o2, x.to(DEV), w13, K().SWIGLU)
        assert err(o2, sw) < 6e-3


@pytest.mark.parametrize("M,F,D", [(3, 48, 72), (40, 160, 96), (70, 16, 40)])
def test_linear_bf16_swiglu_epilogue(M, F, D):
    from lastengine_b200.parts.ffn import fuse_gate_up
    x = gen(M, D, seed=12, dtype=torch.bfloat16)
    w1, w3 = gen(F, D, seed=13, dtype=torch.bfloat16), gen(F, D, seed=14, dtype=torch.bfloat16)
    want = P.silu(x.double() @ w1.double().T) * (x.double() @ w3.double().T)
    w13 = fuse_gate_up(w1, w3, True).to(DEV)
    out = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
    K().linear(out, x.to(DEV), w13, K().SWIGLU, streaming=True)
    assert err(out, want) < 6e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_linear_grouped(dtype):
    E, N, K_ = 5, 40, 56
    counts = [3, 0, 70, 1, 9]
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32)
    Ptot = int(offs[-1])
    x, w = gen(Ptot, K_, seed=15, dtype=dtype), gen(E, N, K_, seed=16, dtype=dtype)
    want = torch.zeros(Ptot, N, dtype=torch.float64)
    for e in range(E):
        a, b = int(offs[e]), int(offs[e + 1])
        want[a:b] = x[a:b].double() @ w[e].double().T
    out = torch.empty(Ptot, N, device=DEV)
    K().linear(out, x.to(DEV), w.to(DEV), group_offsets=offs.to(DEV), rows_hint=Ptot)
    assert err(out, want) < 1e-5


@pytest.mark.parametrize("counts,N,K_", [([3, 0, 0, 1, 9, 0, 2], 48, 72), ([1, 0, 0, 0, 0, 0, 0, 4], 3584, 2048),
                                         ([17, 8, 0, 33, 1, 16, 9, 5], 96, 200), ([5] * 32, 352, 136),
                                         ([0, 0, 0, 0, 0, 0, 0, 0, 0, 7], 64, 64)])
def test_linear_grouped_stream(counts, N, K_):
    """Grouped products through the ring-fed kernel: experts without rows, with one row, with more
    rows than one block of 8 or 16 takes; store, add, both result types, and the SwiGLU epilogue."""
    E = len(counts)
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32)
    Ptot = int(offs[-1])
    assert Ptot <= 16 * E                                   # the sizes this kernel is chosen for
    x, w = gen(Ptot, K_, seed=15, dtype=torch.bfloat16), gen(E, N, K_, seed=16, scale=0.05, dtype=torch.bfloat16)
    want = torch.zeros(Ptot, N, dtype=torch.float64)
    for e in range(E):
        a, b = int(offs[e]), int(offs[e + 1])
        want[a:b] = x[a:b].double() @ w[e].double().T
    out = torch.full((Ptot, N), float("nan"), device=DEV)
    K().linear(out, x.to(DEV), w.to(DEV), group_offsets=offs.to(DEV), rows_hint=Ptot)
    assert err(out, want) < 1e-5
    old = torch.empty(Ptot, N, device=DEV)
    K().linear(old, x.to(DEV), w.to(DEV), group_offsets=offs.to(DEV), rows_hint=Ptot, streaming=True)
    assert err(old, want) < 1e-5                            # the register-fed kernel on the same groups
    ob = torch.empty(Ptot, N, device=DEV, dtype=torch.bfloat16)
    K().linear(ob, x.to(DEV), w.to(DEV), group_offsets=offs.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(Ptot, N, seed=17).to(DEV)
    b0 = base.clone()
    K().linear(base, x.to(DEV), w.to(DEV), K().ACCUMULATE, group_offsets=offs.to(DEV))
    assert err(base, b0.cpu().double() + want) < 1e-5
    if N % 32 == 0:
        from lastengine_b200.parts.ffn import fuse_gate_up
        F = N // 2
        w13 = torch.stack([fuse_gate_up(w[e, :F], w[e, F:], True) for e in range(E)]).to(DEV)
        sw = P.silu(want[:, :F]) * want[:, F:]
        o2 = torch.empty(Ptot, F, device=DEV, dtype=torch.bfloat16)
        K().linear(o2, x.to(DEV), w13, K().SWIGLU, group_offsets=offs.to(DEV))
        assert err(o2, sw) < 6e-3


@pytest.mark.parametrize("counts,N,K_", [([300, 0, 129, 1, 700, 128], 96, 200), ([5, 260, 0, 0, 131], 352, 136),
                                         ([128, 128, 128], 512, 64), ([0, 0, 1000, 0], 3584, 256)])
def test_linear_grouped_tcgen05(counts, N, K_):
    """Grouped products with many rows per expert (prompts) on tcgen05: experts without rows, with
    one row, with rows that end inside a tile (the tile's other rows belong to the next expert and
    must not be written by this one), widths that end inside a weight tile."""
    E = len(counts)
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32)
    Ptot = int(offs[-1])
    assert Ptot > 16 * E
    x, w = gen(Ptot, K_, seed=15, dtype=torch.bfloat16), gen(E, N, K_, seed=16, scale=0.05, dtype=torch.bfloat16)
    want = torch.zeros(Ptot, N, dtype=torch.float64)
    for e in range(E):
        a, b = int(offs[e]), int(offs[e + 1])
        want[a:b] = x[a:b].double() @ w[e].double().T
    out = torch.full((Ptot, N), float("nan"), device=DEV)
    K().linear(out, x.to(DEV), w.to(DEV), group_offsets=offs.to(DEV), rows_hint=Ptot)
    K().check_device_status()
    assert err(out, want) < 2e-5
    ob = torch.empty(Ptot, N, device=DEV, dtype=torch.bfloat16)
    K().linear(ob, x.to(DEV), w.to(DEV), group_offsets=offs.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(Ptot, N, seed=17).to(DEV)
    b0 = base.clone()
    K().linear(base, x.to(DEV), w.to(DEV), K().ACCUMULATE, group_offsets=offs.to(DEV))
    assert err(base, b0.cpu().double() + want) < 2e-5
    if N % 32 == 0:
        from lastengine_b200.parts.ffn import fuse_gate_up
        F = N // 2
        w13 = torch.stack([fuse_gate_up(w[e, :F], w[e, F:], True) for e in range(E)]).to(DEV)
        sw = P.silu(want[:, :F]) * want[:, F:]
        o2 = torch.empty(Ptot, F, device=DEV, dtype=torch.bfloat16)
        K().linear(o2, x.to(DEV), w13, K().SWIGLU, group_offsets=offs.to(DEV))
        assert err(o2, sw) < 6e-3
    K().check_device_status()


# ---- short convolution ---------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("Lc,D", [(3, 72), (4, 130), (2, 64)])
def test_shortconv_with_state(dtype, Lc, D):
    """Three sequences with unequal rows in two consecutive steps, one of them shorter than the
    convolution reaches back; compared with the plain convolution over the joined rows."""
    lens1, lens2 = [1, 5, 2], [3, 1, 1]
    slots = [4, 0, 2]
    w = gen(D, Lc, seed=17)
    bcx_all = [gen(a + b, 3 * D, seed=20 + i, dtype=dtype) for i, (a, b) in enumerate(zip(lens1, lens2))]
    state = torch.full((6, D, Lc - 1), 7.0, device=DEV)   # stale contents of other slots
    for s in slots:
        state[s].zero_()
    bb = builder()
    got = [[] for _ in slots]
    for step, lens in enumerate((lens1, lens2)):
        lo = [0] * 3 if step == 0 else lens1
        rows = torch.cat([bcx_all[i][lo[i]:lo[i] + lens[i]] for i in range(3)]).to(DEV)
        batch = bb.build(slots, [[0] * n for n in lens], lo, [], {})
        y = torch.empty(sum(lens), D, device=DEV, dtype=dtype)
        K().shortconv(y, rows, w.to(DEV), None, state, batch, Lc)
        r0 = 0
        for i, n in enumerate(lens):
            got[i].append(y[r0:r0 + n].float().cpu())
            r0 += n
    for i in range(3):
        bcx = bcx_all[i].double()
        bx = bcx[:, :D] * bcx[:, 2 * D:]
        padded = torch.cat([torch.zeros(Lc - 1, D, dtype=torch.float64), bx])
        acc = sum(padded[j:j + bx.shape[0]] * w.double()[:, j][None] for j in range(Lc))
        want = bcx[:, D:2 * D] * acc
        assert err(torch.cat(got[i]), want) < (1e-6 if dtype == torch.float32 else 5e-3)
        assert err(state[slots[i]].cpu().T, padded[-(Lc - 1):]) < 1e-6      # oldest first
    assert float(state[1].min()) == 7.0 and float(state[5].max()) == 7.0     # other slots untouched


@pytest.mark.parametrize("Lc,D", [(3, 136), (4, 72), (3, 2048)])
def test_shortconv_many_rows(Lc, D):
    """Prompts long enough for the kernel that walks several rows per thread: sequences start in
    the middle of a thread's rows, one is shorter than the filter, one slot is padding, and one
    starts from a state that is not zero."""
    lens = [1, 301, 2, 130, 77]
    slots = [3, 1, -1, 0, 2]
    w = gen(D, Lc, seed=18)
    bcx = [gen(n, 3 * D, seed=40 + i, dtype=torch.bfloat16) for i, n in enumerate(lens)]
    state = torch.zeros(4, D, Lc - 1, device=DEV)
    old = gen(D, Lc - 1, seed=19)
    state[2] = old.to(DEV)
    batch = builder().build(slots, [[0] * n for n in lens], [0, 0, 0, 0, 5], [], {})
    y = torch.full((sum(lens), D), float("nan"), device=DEV, dtype=torch.bfloat16)
    K().shortconv(y, torch.cat(bcx).to(DEV), w.to(DEV), None, state, batch, Lc)
    r0 = 0
    for i, n in enumerate(lens):
        got = y[r0:r0 + n].float().cpu()
        r0 += n
        if slots[i] < 0:
            assert float(got.abs().max()) == 0.0
            continue
        x = bcx[i].double()
        bx = x[:, :D] * x[:, 2 * D:]
        before = old.double().T if slots[i] == 2 else torch.zeros(Lc - 1, D, dtype=torch.float64)
        padded = torch.cat([before, bx])
        acc = sum(padded[j:j + n] * w.double()[:, j][None] for j in range(Lc))
        assert err(got, x[:, D:2 * D] * acc) < 5e-3, i
        assert err(state[slots[i]].cpu().T, padded[-(Lc - 1):]) < 1e-6, i


@pytest.mark.parametrize("B,D,K_,Lc", [(8, 2048, 2048, 3), (1, 72, 40, 2), (13, 136, 200, 4), (16, 48, 64, 5), (5, 100, 72, 3),
                                       (40, 2048, 2048, 3), (100, 136, 1024, 4), (18, 48, 512, 5), (90, 136, 1024, 4)])
def test_shortconv_decode_fused(B, D, K_, Lc):
    """Projection and convolution of a decode step without a convolution kernel (up to 16 sequences:
    one launch; more: the sliced product, whose second kernel convolves), three steps in a row so that the
    state it writes is the state it reads next; one sequence is padding, the slots are not in order
    and other slots hold stale values.  Compared with the plain formulas (projection rounded to
    bfloat16 as the two-kernel path stores it) and with the two-kernel path itself."""
    h_all = [gen(B, K_, seed=60 + t, dtype=torch.bfloat16) for t in range(3)]
    w_in = gen(3 * D, K_, seed=63, scale=0.05, dtype=torch.bfloat16)
    w = gen(D, Lc, seed=64)
    slots = [(5 * i + 3) % (B + 3) for i in range(B)]
    assert len(set(slots)) == B
    if B > 2:
        slots[1] = -1
    state = torch.full((B + 3, D, Lc - 1), 7.0, device=DEV)
    start = gen(B, D, Lc - 1, seed=65)
    for i, s in enumerate(slots):
        if s >= 0:
            state[s] = start[i].to(DEV)
    state2 = state.clone()
    hist = start.double().permute(0, 2, 1).clone()          # [B, Lc-1, D], oldest first
    bb = builder()
    for t in range(3):
        batch = bb.build(slots, [[0]] * B, [t] * B, [], {})
        y = torch.full((B, D), float("nan"), device=DEV, dtype=torch.bfloat16)
        assert K().shortconv_decode_fused(y, h_all[t].to(DEV), w_in.to(DEV), w.to(DEV), None, state, batch, Lc)
        bcx = torch.empty(B, 3 * D, device=DEV, dtype=torch.bfloat16)
        K().linear(bcx, h_all[t].to(DEV), w_in.to(DEV))
        y2 = torch.empty(B, D, device=DEV, dtype=torch.bfloat16)
        K().shortconv(y2, bcx, w.to(DEV), None, state2, batch, Lc)
        p = (h_all[t].double() @ w_in.double().T).to(torch.bfloat16).double()
        bx = p[:, :D] * p[:, 2 * D:]
        taps = torch.cat([hist, bx[:, None]], dim=1)          # [B, Lc, D]
        want = p[:, D:2 * D] * (taps * w.double().T[None]).sum(1)
        hist = taps[:, 1:]
        for i, s in enumerate(slots):
            if s < 0:
                assert float(y[i].abs().max()) == 0.0
                continue
            assert err(y[i], want[i]) < 6e-3, (t, i)
            assert err(y[i], y2[i].float().cpu()) < 6e-3, (t, i)
            assert err(state[s].cpu().T, hist[i]) < 6e-3, (t, i)
    used = [s for s in slots if s >= 0]
    for s in range(B + 3):
        if s not in used:
            assert float(state[s].min()) == 7.0 and float(state[s].max()) == 7.0


@pytest.mark.parametrize("M,D,K_,N2", [(8, 2048, 2048, 6144), (1, 72, 40, 64), (13, 136, 200, 96), (16, 104, 64, 32),
                                       (64, 2048, 5632, 6144), (17, 72, 40, 64), (100, 136, 200, 96), (128, 104, 64, 32),
                                       (80, 2048, 5632, 6144), (96, 136, 200, 96)])
def test_norm_split_between_two_products(M, D, K_, N2):
    """An RMSNorm split between the product that adds into the residual and the product that reads
    the normed rows (decode steps): the first leaves bfloat16(x * g) and partial sums of x^2, the
    second scales its sums by rsqrt(mean + eps).  Up to 16 rows through the weight stream, above
    through the sliced tcgen05 product.  Compared with norm and products in float64."""
    from lastengine_b200.parts.ffn import fuse_gate_up
    eps = 3e-5
    a, w = gen(M, K_, seed=70, dtype=torch.bfloat16), gen(D, K_, seed=71, scale=0.05, dtype=torch.bfloat16)
    x0, g = gen(M, D, seed=72, scale=3.0), 1.0 + gen(D, seed=73, scale=0.3)
    x = x0.to(DEV)
    sp = K().SplitNorm(torch.empty(M, D, device=DEV, dtype=torch.bfloat16),
                       torch.full((M, -(-D // 16)), float("nan"), device=DEV), g.to(DEV), eps)
    K().linear(x, a.to(DEV), w.to(DEV), K().ACCUMULATE, emit=sp)
    assert sp.filled
    xn = x0.double() + a.double() @ w.double().T
    assert err(x, xn) < 2e-5
    assert err(sp.values, xn * g.double()) < 5e-3
    assert err(sp.ssq.sum(1), (xn ** 2).sum(1)) < 1e-5
    normed = xn * torch.rsqrt((xn ** 2).mean(1, keepdim=True) + eps) * g.double()
    w2 = gen(N2, D, seed=74, scale=0.05, dtype=torch.bfloat16)
    out = torch.empty(M, N2, device=DEV, dtype=torch.bfloat16)
    K().linear(out, sp.values, w2.to(DEV), scale=sp)
    assert err(out, normed @ w2.double().T) < 6e-3
    F = N2 // 2
    o2 = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
    K().linear(o2, sp.values, fuse_gate_up(w2[:F], w2[F:], True).to(DEV), K().SWIGLU, scale=sp)
    assert err(o2, P.silu(normed @ w2[:F].double().T) * (normed @ w2[F:].double().T)) < 6e-3
    K().check_device_status()


# ---- rotation and cache write ---------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,rope_dim,lens", [(4, 2, 16, 16, [3, 70]), (3, 1, 48, 32, [3, 70]), (5, 5, 80, 80, [3, 70]),
                                                      (2, 1, 64, 64, [3, 70]), (6, 2, 128, 128, [3, 70]),
                                                      (9, 3, 64, 64, [60, 100]), (13, 1, 64, 64, [400, 290])])
def test_qk_rope_store(dtype, nh, nkv, hd, rope_dim, lens):
    if dtype == torch.float32 and max(lens) > 128:
        # a float angle is off by up to position x 6e-8: the float path is compared at short positions
        # only; the long case is there for the bfloat16 kernel that takes several heads per warp
        lens = [n // 4 for n in lens]
    page = 64
    pos0 = [62, 5]                                  # rows cross a page boundary
    M = sum(lens)
    width = nh * hd + 2 * nkv * hd
    qkv = gen(M, width, seed=30, dtype=dtype)
    qn, kn = 1 + 0.1 * gen(hd, seed=31), 1 + 0.1 * gen(hd, seed=32)
    theta, eps = 12345.0, 1e-4
    inv = torch.pow(torch.tensor(theta, dtype=torch.float64), -2.0 * torch.arange(rope_dim // 2, dtype=torch.float64) / rope_dim).float()
    width = max(-(-(p + n) // page) for p, n in zip(pos0, lens))
    n_pages = 2 * width + 2
    order = np.random.default_rng(5).permutation(n_pages)[:2 * width].astype(np.int32)   # pages in no order
    tables = {0: order.reshape(2, width)}
    kp = torch.zeros(n_pages, nkv, page, hd, device=DEV, dtype=dtype)
    vp = torch.zeros(n_pages, nkv, hd, page, device=DEV, dtype=dtype)      # values: positions contiguous
    batch = builder().build([0, 1], [[0] * n for n in lens], pos0, [], tables)
    q_out = torch.empty(M, nh * hd, device=DEV, dtype=dtype)
    qd = qkv.to(DEV)
    K().qk_rope_store(q_out, qd[:, :nh * hd], qd[:, nh * hd:(nh + nkv) * hd], qd[:, (nh + nkv) * hd:], kp, vp,
                      batch.tables[0], batch, qn.to(DEV), kn.to(DEV), eps, inv.to(DEV), rope_dim, True, nh, nkv, hd, page)
    tol = 1e-5 if dtype == torch.float32 else 6e-3
    r0 = 0
    for b, n in enumerate(lens):
        rows = qkv[r0:r0 + n].double()
        pos = torch.arange(pos0[b], pos0[b] + n)
        q = P.rope(P.rms_norm(rows[:, :nh * hd].view(n, nh, hd), qn.double(), eps), pos, rope_dim, theta)
        k = P.rope(P.rms_norm(rows[:, nh * hd:(nh + nkv) * hd].view(n, nkv, hd), kn.double(), eps), pos, rope_dim, theta)
        v = rows[:, (nh + nkv) * hd:].view(n, nkv, hd)
        assert err(q_out[r0:r0 + n].view(n, nh, hd), q) < tol
        for i, p_ in enumerate(pos.tolist()):
            pg = int(tables[0][b, p_ // page])
            assert err(kp[pg, :, p_ % page, :], k[i]) < tol
            assert err(vp[pg, :, :, p_ % page], v[i]) < tol
        r0 += n


@pytest.mark.parametrize("lens,nh,nkv,weights,rotate", [([128], 4, 2, True, True), ([60, 69], 5, 5, True, True),
                                                        ([1, 200, 3], 32, 8, True, True), ([700, 485], 8, 2, True, True),
                                                        ([129], 3, 1, False, True), ([130], 4, 4, True, False)])
def test_qk_rope_store_of_many_rows_gives_the_bits_of_few(lens, nh, nkv, weights, rotate):
    """Steps of 128 rows and more (blocks of two rows, from 8 rows an SM on of eight) against the same rows in steps of at most
    60: q, the cached keys and the cached values, bit for bit.  Odd lengths, starts off the multiples of eight (values leave
    in single numbers there and in runs of eight elsewhere), a padding sequence in front."""
    hd, page, eps = 64, 64, 1e-4
    M = sum(lens)
    qkv = gen(M, (nh + 2 * nkv) * hd, seed=30, dtype=torch.bfloat16).to(DEV)
    qn, kn = ((1 + 0.1 * gen(hd, seed=31)).to(DEV), (1 + 0.1 * gen(hd, seed=32)).to(DEV)) if weights else (None, None)
    inv = torch.pow(torch.tensor(12345.0, dtype=torch.float64), -torch.arange(32, dtype=torch.float64) / 32).float().to(DEV) \
        if rotate else None
    pos0 = [0, 62, 5][:len(lens)]
    slots = [-1, 0, 1] if len(lens) == 3 else list(range(len(lens)))
    width = max(-(-(p + n) // page) for p, n in zip(pos0, lens))
    n_pages = len(lens) * width + 1
    table = np.random.default_rng(5).permutation(n_pages)[:len(lens) * width].astype(np.int32).reshape(len(lens), width)

    def run(pieces):
        """pieces: [(sequence, first row, rows)] per step"""
        kp = torch.zeros(n_pages, nkv, page, hd, device=DEV, dtype=torch.bfloat16)
        vp = torch.zeros(n_pages, nkv, hd, page, device=DEV, dtype=torch.bfloat16)
        out = torch.zeros(M, nh * hd, device=DEV, dtype=torch.bfloat16)
        for step in pieces:
            lo = sum(lens[:step[0][0]]) + step[0][1]
            n = sum(c for _, _, c in step)
            batch = builder().build([slots[b] for b, _, _ in step], [[0] * c for _, _, c in step],
                                    [pos0[b] + f for b, f, _ in step], [], {0: table[[b for b, _, _ in step]]})
            r = qkv[lo:lo + n]
            K().qk_rope_store(out[lo:lo + n], r[:, :nh * hd], r[:, nh * hd:(nh + nkv) * hd], r[:, (nh + nkv) * hd:], kp, vp,
                              batch.tables[0], batch, qn, kn, eps, inv, hd if rotate else 0, True, nh, nkv, hd, page,
                              **({} if rotate else {"temperature": (0.3, 7.0)}))
        return out, kp, vp

    whole = run([[(b, 0, n) for b, n in enumerate(lens)]])
    parts = run([[(b, f, min(60, n - f))] for b, n in enumerate(lens) for f in range(0, n, 60)])
    for a, b in zip(whole, parts):
        assert torch.equal(a, b)


@pytest.mark.parametrize("M,nh", [(600, 32), (520, 32), (190, 8), (2100, 8)])
def test_rotation_of_queries_alone_on_both_sides_of_its_line(M, nh):
    """Queries without keys: from 16,384 of them on the kernel of many rows, below it the lanes; the bits of steps of 60 rows."""
    q = gen(M, nh * 64, seed=30, dtype=torch.bfloat16).to(DEV)
    qn = (1 + 0.1 * gen(64, seed=31)).to(DEV)
    inv = torch.pow(torch.tensor(12345.0, dtype=torch.float64), -torch.arange(32, dtype=torch.float64) / 32).float().to(DEV)
    table = {0: np.arange(-(-M // 64), dtype=np.int32)[None]}

    def run(step):
        out = torch.zeros(M, nh * 64, device=DEV, dtype=torch.bfloat16)
        for lo in range(0, M, step):
            n = min(step, M - lo)
            b = builder().build([0], [[0] * n], [lo], [], table)
            K().qk_rope_store(out[lo:lo + n], q[lo:lo + n], None, None, None, None, b.tables[0], b, qn, None, 1e-4, inv, 64, True, nh,
                              1, 64, 64)
        return out

    assert torch.equal(run(M), run(60))


# ---- words between host and device ---------------------------------------------------------------------
def test_words_of_dropped_owners_stay_until_the_device_is_through_with_them():
    """Builders and result buffers dropped while their transfers wait behind other work: every step finds its own words, and
    what a late transfer brings to the host lands in no other owner's buffer."""
    dev = torch.device(DEV)
    torch.cuda._sleep(100_000_000)
    steps = [builder().build([0], [list(range(100 * i, 100 * i + 40))], [i], [39], {}) for i in range(20)]
    for i in range(4):
        w = K().PinnedWords(1025, dev)
        K().stage_words(w.words, torch.full((1025,), i, dtype=torch.int32, device=DEV), 1025)
        w.mark()
    del w
    mine = [K().PinnedWords(1025, dev) for _ in range(4)]
    for m in mine:
        m.words.fill_(-1)
    torch.cuda.synchronize()
    for i, b in enumerate(steps):
        assert b.tokens.tolist() == list(range(100 * i, 100 * i + 40)) and b.row_pos.tolist() == list(range(i, i + 40))
    assert all(bool((m.words == -1).all()) for m in mine)


@pytest.mark.parametrize("replayed", [False, True])
def test_steps_are_brought_by_a_kernel_only_where_a_graph_follows(replayed):
    """Behind the copy engine any kernel may start; behind a kernel of ours the next one could start before its words are
    visible, unless a graph's launch stands between."""
    from lastengine_b200.engine.batch import BatchBuilder
    b = BatchBuilder(torch.device(DEV), replayed=replayed)
    n = K().launch_count()
    step = b.build([0], [[5, 6, 7]], [2], [2], {})
    assert K().launch_count() - n == int(replayed)
    assert step.tokens.tolist() == [5, 6, 7] and step.row_pos.tolist() == [2, 3, 4]
    b.host_view("tokens")[:] = [8, 9, 10]
    b.resend()
    assert K().launch_count() - n == 2 * int(replayed)
    assert step.tokens.tolist() == [8, 9, 10]


@pytest.mark.parametrize("n", [1, 3, 255, 256, 257, 4095, 4096, 4097])
def test_stage_words_both_ways(n):
    """Up to 4,096 words by a kernel (of 256 or 1,024 threads), more by a copy: all of them arrive and nothing beyond them."""
    dev = torch.device(DEV)
    host, back = K().PinnedWords(5000, dev), K().PinnedWords(5000, dev)
    host.words.copy_(torch.arange(5000, dtype=torch.int32) * 7 - 3)
    back.words.fill_(-9)
    d = torch.full((5000,), -5, dtype=torch.int32, device=DEV)
    K().stage_words(d, host.words, n)
    host.mark()
    K().stage_words(back.words, d, n)
    back.mark()
    back.wait()
    assert torch.equal(back.words[:n], host.words[:n]) and bool((back.words[n:] == -9).all())
    assert bool((d[n:] == -5).all())


# ---- attention ---------------------------------------------------------------------------------------
def plain_attention(q, k, v, qpos, window, scale):
    """q [Tq, nh, hd], k/v [Tk, nkv, hd] (positions 0..Tk-1), qpos [Tq]."""
    Tq, nh, hd = q.shape
    nkv = k.shape[1]
    out = torch.zeros_like(q)
    t = torch.arange(k.shape[0])
    for h in range(nh):
        s = (q[:, h] @ k[:, h // (nh // nkv)].T) * scale
        ok = t[None] <= qpos[:, None]
        if window > 0:
            ok &= t[None] > qpos[:, None] - window
        s = s.masked_fill(~ok, float("-inf"))
        out[:, h] = torch.softmax(s, -1) @ v[:, h // (nh // nkv)]
    return out


def fill_cache(k, v, pages, nkv, hd, page, dtype):
    n_pages = max(pages) + 2
    kp = torch.full((n_pages, nkv, page, hd), float("nan"), dtype=dtype)   # unused places hold NaN
    vp = torch.full((n_pages, nkv, hd, page), float("nan"), dtype=dtype)   # values: positions contiguous
    for t in range(k.shape[0]):
        kp[pages[t // page], :, t % page] = k[t].to(dtype)
        vp[pages[t // page], :, :, t % page] = v[t].to(dtype)
    return kp.to(DEV), vp.to(DEV)


@pytest.mark.parametrize("nh,nkv,hd", [(32, 8, 64), (6, 2, 128), (5, 5, 64), (16, 1, 64)])
@pytest.mark.parametrize("window,gated,with_norm", [(0, False, True), (40, True, True), (0, False, False)])
def test_decode_attention_that_norms_rotates_and_stores_the_step_itself(nh, nkv, hd, window, gated, with_norm):
    """A decode step handed to the attention kernel as the projection left it (raw q, k and v) against
    the same step with the rotary kernel first: the same output bits and the same cache, at every
    split count, for sequences whose new position starts a page, ends one, or is the first of all;
    a padding sequence among them; and against double-precision arithmetic."""
    page, dtype = 64, torch.bfloat16
    lens = [130, 1, 64, 65, 257, 7]                 # lengths after the step: the new token sits at len - 1
    slots = [0, 1, -1, 2, 3, 4]
    B = len(lens)
    width = max(-(-n // page) for n in lens)
    n_pages = B * width + 1
    order = np.random.default_rng(6).permutation(n_pages)[:B * width].astype(np.int32).reshape(B, width)
    kp0 = gen(n_pages, nkv, page, hd, seed=50, dtype=dtype).to(DEV)
    vp0 = gen(n_pages, nkv, hd, page, seed=51, dtype=dtype).to(DEV)
    qkv = gen(B, (nh + 2 * nkv) * hd + nh, seed=52, dtype=dtype).to(DEV)        # q | k | v | gate as one projection
    q_in, k_in = qkv[:, :nh * hd], qkv[:, nh * hd:(nh + nkv) * hd]
    v_in, gate = qkv[:, (nh + nkv) * hd:(nh + 2 * nkv) * hd], (qkv[:, (nh + 2 * nkv) * hd:] if gated else None)
    qn = (1 + 0.1 * gen(hd, seed=53)).to(DEV) if with_norm else None
    kn = (1 + 0.1 * gen(hd, seed=54)).to(DEV) if with_norm else None
    theta, eps, scale = 5e4, 1e-5, 1 / math.sqrt(hd)
    inv = torch.pow(torch.tensor(theta, dtype=torch.float64), -2.0 * torch.arange(hd // 2, dtype=torch.float64) / hd).float().to(DEV)
    batch = builder().build(slots, [[0]] * B, [n - 1 for n in lens], [], {0: order})
    assert K().decode_attention_takes_raw(dtype, batch, B, nh, nkv, hd, page, inv, hd, True)
    for splits in (1, 2, 5):
        scratch = torch.empty(B * nh * splits * (hd + 2), device=DEV)
        # the two-kernel way
        kp_a, vp_a = kp0.clone(), vp0.clone()
        q_rot = torch.empty(B, nh * hd, device=DEV, dtype=dtype)
        K().qk_rope_store(q_rot, q_in, k_in, v_in, kp_a, vp_a, batch.tables[0], batch, qn, kn, eps, inv, hd, True, nh, nkv, hd, page)
        want = torch.empty(B, nh * hd, device=DEV, dtype=dtype)
        K().attention(want, q_rot, kp_a, vp_a, batch.tables[0], batch, nh, nkv, hd, page, window, scale, gate=gate,
                      n_splits=splits, scratch=scratch)
        # the kernel that does it all
        kp_b, vp_b = kp0.clone(), vp0.clone()
        got = torch.full_like(want, float("nan"))
        K().attention(got, None, kp_b, vp_b, batch.tables[0], batch, nh, nkv, hd, page, window, scale, gate=gate,
                      n_splits=splits, scratch=scratch, raw=K().RawQKV(q_in, k_in, v_in, qn, kn, eps, inv, hd, True))
        torch.cuda.synchronize()
        assert torch.equal(kp_a, kp_b) and torch.equal(vp_a, vp_b), f"{splits} splits: the caches differ"
        assert not torch.equal(kp_a, kp0)
        assert torch.equal(got, want), f"{splits} splits: {err(got, want):.3e}"
    # against double precision, from the cache the kernel left
    for b, n in enumerate(lens):
        if slots[b] < 0:
            assert float(got[b].float().abs().max()) == 0.0
            continue
        k = torch.stack([kp_b[int(order[b, t // page]), :, t % page].double().cpu() for t in range(n)])
        v = torch.stack([vp_b[int(order[b, t // page]), :, :, t % page].double().cpu() for t in range(n)])
        row = qkv[b].double().cpu()
        q = row[:nh * hd].view(1, nh, hd)
        if with_norm:
            q = P.rms_norm(q, qn.double().cpu(), eps)
        q = P.round_bf16(P.rope(q, torch.tensor([n - 1]), hd, theta))
        o = plain_attention(q, k, v, torch.tensor([n - 1]), window, scale)[0]
        if gated:
            o = o * torch.sigmoid(row[(nh + 2 * nkv) * hd:])[:, None]
        assert err(got[b].view(nh, hd), o) < 8e-3, b
        # the new key is the normed and rotated one
        kn_new = row[nh * hd:(nh + nkv) * hd].view(1, nkv, hd)
        if with_norm:
            kn_new = P.rms_norm(kn_new, kn.double().cpu(), eps)
        assert err(k[n - 1], P.rope(kn_new, torch.tensor([n - 1]), hd, theta)[0]) < 6e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 16), (3, 1, 48), (10, 5, 80), (16, 1, 32), (8, 8, 128), (32, 8, 64), (12, 2, 96)])
@pytest.mark.parametrize("window", [0, 40])
def test_attention_prompt_and_decode(dtype, nh, nkv, hd, window):
    page, Tk = 64, 150
    k, v = gen(Tk, nkv, hd, seed=40, dtype=dtype), gen(Tk, nkv, hd, seed=41, dtype=dtype)
    pages = [3, 0, 5]
    kp, vp = fill_cache(k, v, pages, nkv, hd, page, dtype)
    scale = 1 / math.sqrt(hd)
    tol = 2e-5 if dtype == torch.float32 else 8e-3
    tables = {0: np.array([pages], dtype=np.int32)}
    # a chunk of 37 rows continuing at position 100, then a single row at the end, split four ways
    for q0, n, splits in ((100, 37, 1), (0, 150, 1), (149, 1, 1), (149, 1, 4), (70, 1, 16)):
        q = gen(n, nh, hd, seed=42 + n, dtype=dtype)
        batch = builder().build([0], [[0] * n], [q0], [], tables)
        out = torch.empty(n, nh * hd, device=DEV, dtype=dtype)
        scratch = torch.empty(n * nh * splits * (hd + 2), device=DEV) if splits > 1 else None
        K().attention(out, q.reshape(n, nh * hd).to(DEV), kp, vp, batch.tables[0], batch, nh, nkv, hd, page,
                      window, scale, n_splits=splits, scratch=scratch)
        want = plain_attention(q.double(), k.double(), v.double(), torch.arange(q0, q0 + n), window, scale)
        assert err(out.view(n, nh, hd), want) < tol, (q0, n, splits)


@pytest.mark.parametrize("nh,nkv,hd", [(4, 2, 64), (3, 1, 20), (16, 2, 128)])
@pytest.mark.parametrize("window", [0, 40])
def test_general_attention_loads_16_bytes_or_single_numbers(nh, nkv, hd, window):
    """32-bit caches on 16-byte addresses (four numbers a load) and off them (single numbers): the same bits, for a prompt, a
    continued one and a step of one row whole and in splits; unused places of the pages hold NaN."""
    page, Tk, pages = 64, 150, [3, 0, 5]
    k, v = gen(Tk, nkv, hd, seed=40), gen(Tk, nkv, hd, seed=41)
    kp, vp = fill_cache(k, v, pages, nkv, hd, page, torch.float32)

    def off(t):
        b = torch.empty(t.numel() + 1, device=DEV)
        b[1:] = t.reshape(-1)
        return b[1:].view(t.shape)

    assert kp.data_ptr() % 16 == 0 and off(kp).data_ptr() % 16 == 4
    for q0, n, splits in ((0, 150, 1), (100, 37, 1), (149, 1, 1), (149, 1, 4)):
        q = gen(n, nh * hd, seed=42 + n).to(DEV)
        batch = builder().build([0], [[0] * n], [q0], [], {0: np.array([pages], dtype=np.int32)})
        got = []
        for a, b in ((kp, vp), (off(kp), off(vp)), (kp, off(vp))):
            out = torch.full((n, nh * hd), float("nan"), device=DEV)
            scratch = torch.empty(n * nh * splits * (hd + 2), device=DEV) if splits > 1 else None
            K().attention(out, q, a, b, batch.tables[0], batch, nh, nkv, hd, page, window, hd ** -0.5, n_splits=splits, scratch=scratch)
            got.append(out)
        assert bool(got[0].isfinite().all()) and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])


@pytest.mark.parametrize("dtype,nh,nkv,hd", [(torch.float32, 4, 4, 64), (torch.float32, 8, 2, 64), (torch.float32, 3, 1, 48),
                                             (torch.bfloat16, 4, 4, 48)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("window", [0, 40])
def test_values_of_tiles_a_row_does_not_read_do_not_reach_it(dtype, nh, nkv, hd, bad, window):
    """The general kernel takes rows of several positions through a tile of 32 keys together.  A value that is not finite, at
    the last position (of a tile of its own) or at one that a window has left behind, must stay out of the rows whose
    tiles it does not lie in."""
    page, Tk = 64, 97
    k, v = gen(Tk, nkv, hd, seed=60, dtype=dtype), gen(Tk, nkv, hd, seed=61, dtype=dtype)
    q = gen(Tk, nh, hd, seed=62, dtype=dtype)
    tables = {0: np.array([[1, 0]], dtype=np.int32)}
    scale = 1 / math.sqrt(hd)
    want = plain_attention(q.double(), k.double(), v.double(), torch.arange(Tk), window, scale)
    batch = builder().build([0], [[0] * Tk], [0], [], tables)
    # position 96 lies in the tile from 96 on, which rows below 96 do not read; position 0 in the first tile, which rows from
    # 71 on (71 - 40 + 1 = 32) do not read through the window
    for at, clean in ((Tk - 1, slice(0, 96)), (0, slice(71, Tk) if window else slice(0, 0))):
        w = v.clone()
        w[at] = bad
        kp, vp = fill_cache(k, w, [1, 0], nkv, hd, page, dtype)
        out = torch.zeros(Tk, nh * hd, device=DEV, dtype=dtype)
        K().attention(out, q.reshape(Tk, nh * hd).to(DEV), kp, vp, batch.tables[0], batch, nh, nkv, hd, page, window, scale)
        got = out.view(Tk, nh, hd)[clean]
        assert bool(got.isfinite().all())
        assert clean.stop == 0 or err(got, want[clean]) < (2e-5 if dtype == torch.float32 else 8e-3)
        assert not bool(out.view(Tk, nh, hd)[at].isfinite().any())      # ... and reaches the row whose own it is


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_far_key_and_window_edge(dtype):
    """One early key is made to dominate: among hundreds of keys the output must be its value;
    with a window that ends just before it, it must vanish, and one position earlier it must not."""
    nh, nkv, hd, page, Tk = 4, 2, 64, 64, 300
    k, v = gen(Tk, nkv, hd, seed=50, scale=0.1), gen(Tk, nkv, hd, seed=51)
    q = gen(1, nh, hd, seed=52, scale=0.1)
    far = 3
    k[far] = 0
    k[far, :, 0] = 40.0
    q[..., 0] = 40.0                       # score 1600/8 = 200 against O(1) elsewhere
    k, v, q = k.to(dtype), v.to(dtype), q.to(dtype)
    pages = [1, 4, 2, 0, 6]
    kp, vp = fill_cache(k, v, pages, nkv, hd, page, dtype)
    tables = {0: np.array([pages], dtype=np.int32)}
    scale = 1 / math.sqrt(hd)
    for splits in (1, 5):
        for window, sees in ((0, True), (Tk - far, True), (Tk - far - 1, False)):
            batch = builder().build([0], [[0]], [Tk - 1], [], tables)
            out = torch.empty(1, nh * hd, device=DEV, dtype=dtype)
            scratch = torch.empty(nh * splits * (hd + 2), device=DEV)
            K().attention(out, q.reshape(1, nh * hd).to(DEV), kp, vp, batch.tables[0], batch, nh, nkv, hd, page,
                          window, scale, n_splits=splits, scratch=scratch)
            want = plain_attention(q.double(), k.double(), v.double(), torch.tensor([Tk - 1]), window, scale)
            assert err(out.view(1, nh, hd), want) < (2e-5 if dtype == torch.float32 else 8e-3)
            hit = err(out.view(1, nh, hd)[0, 0], v[far, 0].double()) < 1e-2
            assert hit == sees, (splits, window)


@pytest.mark.parametrize("nh,nkv", [(4, 4), (4, 2), (8, 2), (8, 1)])
@pytest.mark.parametrize("window", [0, 150])
def test_attention_long_prompts_on_tcgen05(nh, nkv, window):
    """Head size 64 with 1, 2, 4 and 8 query heads per kv head: the tcgen05 prompt kernel.  Two
    sequences of several tiles and pages; the second continues at a position that is no multiple
    of anything.  Keys grow along the sequence, so every row's maximum moves many times by more
    than the factor the kernel tolerates before it rescales; one early key dominates a late query;
    unused places of the cache hold NaN."""
    hd, page, dtype = 64, 64, torch.bfloat16
    lens_k, pos0, qn = [700, 333], [0, 203], [700, 130]
    ks = [gen(n, nkv, hd, seed=160 + i) * torch.linspace(0.2, 3.0, n)[:, None, None] for i, n in enumerate(lens_k)]
    vs = [gen(n, nkv, hd, seed=170 + i) for i, n in enumerate(lens_k)]
    qs = [gen(n, nh, hd, seed=180 + i) for i, n in enumerate(qn)]
    far = 5
    ks[0][far] = 0
    ks[0][far, :, 0] = 60.0
    qs[0][650, :, :] = 0
    qs[0][650, :, 0] = 8.0                       # score 480/8 = 60 against a few elsewhere
    ks, vs, qs = [t.to(dtype) for t in ks], [t.to(dtype) for t in vs], [t.to(dtype) for t in qs]
    n_pages = 20
    order = np.random.default_rng(7).permutation(n_pages).astype(np.int32)
    page_lists = [order[:11].tolist(), order[11:17].tolist()]
    pools_k = torch.full((n_pages, nkv, page, hd), float("nan"), dtype=dtype)
    pools_v = torch.full((n_pages, nkv, hd, page), float("nan"), dtype=dtype)
    for i in range(2):
        for t in range(lens_k[i]):
            pools_k[page_lists[i][t // page], :, t % page] = ks[i][t]
            pools_v[page_lists[i][t // page], :, :, t % page] = vs[i][t]
    table = np.full((2, 11), -1, dtype=np.int32)
    for i, pl in enumerate(page_lists):
        table[i, :len(pl)] = pl
    batch = builder().build([0, 1], [[0] * n for n in qn], pos0, [], {0: table})
    M = sum(qn)
    out = torch.full((M, nh * hd), float("nan"), device=DEV, dtype=dtype)
    K().attention(out, torch.cat(qs).reshape(M, nh * hd).to(DEV), pools_k.to(DEV), pools_v.to(DEV), batch.tables[0],
                  batch, nh, nkv, hd, page, window, 0.125)
    K().check_device_status()
    r0 = 0
    for i, n in enumerate(qn):
        want = plain_attention(qs[i].double(), ks[i].double(), vs[i].double(), torch.arange(pos0[i], pos0[i] + n), window, 0.125)
        assert err(out[r0:r0 + n].view(n, nh, hd), want) < 8e-3, i
        r0 += n
    if window == 0:
        assert err(out[650].view(nh, hd)[0], vs[0][far, 0].double()) < 1e-2     # the far key's value, alone


@pytest.mark.parametrize("nh,nkv,window", [(8, 8, 0), (16, 8, 0), (32, 8, 0), (32, 8, 100), (64, 8, 0)])
def test_prompt_attention_of_few_tiles_gives_the_bits_of_many(nh, nkv, window):
    """Steps of few tiles run two blocks an SM with two buffers of scores, others three with one: a prompt alone and among others."""
    hd, page, n, width, B = 64, 64, 333, 6, 40
    table = np.random.default_rng(12).permutation(B * width).astype(np.int32).reshape(B, width)
    pk, pv = (gen(B * width, nkv, page, hd, seed=s, dtype=torch.bfloat16).to(DEV) for s in (395, 396))
    q = gen(B * n, nh * hd, seed=397, dtype=torch.bfloat16).to(DEV)
    # beyond 2.5 tiles an SM for sure (40 prompts), and for sure not (one): 333 rows are 3 tiles of 128 and more, times 8 heads
    assert B * 3 * nkv > 2.5 * 160 and -(-n * (nh // nkv) // 128) * nkv <= 2.5 * 132

    def run(seqs):
        batch = builder().build(list(range(len(seqs))), [[0] * n] * len(seqs), [0] * len(seqs), [], {0: table[seqs]})
        out = torch.empty(len(seqs) * n, nh * hd, device=DEV, dtype=torch.bfloat16)
        rows = torch.cat([q[i * n:(i + 1) * n] for i in seqs])
        K().attention(out, rows, pk, pv, batch.tables[0], batch, nh, nkv, hd, page, window, 0.125)
        K().check_device_status()
        return out

    many = run(list(range(B)))
    for i in (0, 17, 39):
        assert torch.equal(run([i]), many[i * n:(i + 1) * n])


@pytest.mark.parametrize("nh,nkv", [(4, 4), (4, 2), (8, 2), (8, 1)])
@pytest.mark.parametrize("gate", ["none", "head", "number", "number, unaligned"])
@pytest.mark.parametrize("wide", [False, True])
def test_prompt_attention_of_part_tiles_with_gates(nh, nkv, gate, wide):
    """Last tiles whose warps hold rows of the sequence beside rows beyond it (1 to 127 of 128), which part ways before
    the second half of a row is read from tensor memory; with every form of the output gate, whose 16-byte loads are a
    branch of their own.  Results are bfloat16 and weights one or two bfloat16 terms: the tolerance of the other prompts."""
    hd, page, dtype = 64, 64, torch.bfloat16
    lens = [2, 33, 70, 131, 45]
    width, M = 3, sum(lens)
    table = np.random.default_rng(11).permutation(len(lens) * width).astype(np.int32).reshape(len(lens), width)
    pk = torch.full((table.size, nkv, page, hd), float("nan"), dtype=dtype)
    pv = torch.full((table.size, nkv, hd, page), float("nan"), dtype=dtype)
    q = gen(M, nh, hd, seed=190, dtype=dtype)
    want, r0 = [], 0
    width_g = 0 if gate == "none" else nh if gate == "head" else nh * hd
    g_all = gen(M, width_g + 8, seed=191, dtype=dtype)
    off = 3 if gate.endswith("unaligned") else 0
    g = g_all[:, off:off + width_g]
    for b, n in enumerate(lens):
        k, v = gen(n, nkv, hd, seed=192 + b, dtype=dtype), gen(n, nkv, hd, seed=292 + b, dtype=dtype)
        for t in range(n):
            pk[table[b, t // page], :, t % page] = k[t]
            pv[table[b, t // page], :, :, t % page] = v[t]
        w = plain_attention(q[r0:r0 + n].double(), k.double(), v.double(), torch.arange(n), 0, 0.125)
        if width_g:
            w = w * torch.sigmoid(g[r0:r0 + n].double()).reshape(n, nh, -1)
        want.append(w)
        r0 += n
    batch = builder().build(list(range(len(lens))), [[0] * n for n in lens], [0] * len(lens), [], {0: table})
    out = torch.full((M + 1, nh * hd), float("nan"), device=DEV, dtype=dtype)
    K().attention(out[:M], q.reshape(M, nh * hd).to(DEV), pk.to(DEV), pv.to(DEV), batch.tables[0], batch, nh, nkv, hd, page, 0,
                  0.125, gate=g_all.to(DEV)[:, off:off + width_g] if width_g else None, wide=wide)
    K().check_device_status()
    assert err(out[:M].view(M, nh, hd), torch.cat(want)) < 8e-3
    assert bool(out[M].isnan().all())


@pytest.mark.parametrize("dtype,nh,nkv,hd", [(torch.float32, 6, 2, 48), (torch.bfloat16, 6, 2, 64), (torch.bfloat16, 6, 2, 48),
                                             (torch.bfloat16, 8, 2, 64), (torch.bfloat16, 8, 1, 64)])
def test_attention_batch_of_unequal_sequences(dtype, nh, nkv, hd):
    """Several sequences in one launch, each with its own pages, lengths and row counts; one is padding."""
    page = 64
    lens_k, pos0, qn = [90, 10, 130], [60, 0, 129], [30, 10, 1]
    ks = [gen(n, nkv, hd, seed=60 + i, dtype=dtype) for i, n in enumerate(lens_k)]
    vs = [gen(n, nkv, hd, seed=70 + i, dtype=dtype) for i, n in enumerate(lens_k)]
    pools_k = torch.full((12, nkv, page, hd), float("nan"), dtype=dtype)
    pools_v = torch.full((12, nkv, hd, page), float("nan"), dtype=dtype)
    page_lists = [[7, 2], [9], [0, 11, 4]]
    for i in range(3):
        for t in range(lens_k[i]):
            pools_k[page_lists[i][t // page], :, t % page] = ks[i][t]
            pools_v[page_lists[i][t // page], :, :, t % page] = vs[i][t]
    table = np.full((4, 3), -1, dtype=np.int32)
    for i, pl in enumerate(page_lists):
        table[i if i < 2 else 3, :len(pl)] = pl
    slots, rows = [0, 1, -1, 2], [qn[0], qn[1], 2, qn[2]]
    qs = [gen(n, nh, hd, seed=80 + i, dtype=dtype) for i, n in enumerate(rows)]
    batch = builder().build(slots, [[0] * n for n in rows], [pos0[0], pos0[1], 0, pos0[2]], [], {0: table})
    M = sum(rows)
    out = torch.empty(M, nh * hd, device=DEV, dtype=dtype)
    K().attention(out, torch.cat(qs).reshape(M, nh * hd).to(DEV), pools_k.to(DEV), pools_v.to(DEV), batch.tables[0],
                  batch, nh, nkv, hd, page, 0, 0.2)
    r0 = 0
    for j, (s, n) in enumerate(zip(slots, rows)):
        if s >= 0:
            p0 = [pos0[0], pos0[1], 0, pos0[2]][j]
            want = plain_attention(qs[j].double(), ks[s].double(), vs[s].double(), torch.arange(p0, p0 + n), 0, 0.2)
            assert err(out[r0:r0 + n].view(n, nh, hd), want) < (2e-5 if dtype == torch.float32 else 8e-3)
        else:
            assert float(out[r0:r0 + n].abs().max()) == 0.0
        r0 += n


# ---- experts ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,k,norm,bias,scaling", [(8, 2, True, True, 1.0), (5, 1, False, False, 1.5), (32, 4, True, True, 2.0)])
def test_moe_router_align_combine(dtype, E, k, norm, bias, scaling):
    M, D = 77, 104
    h = gen(M, D, seed=90, dtype=dtype)
    wr, b = gen(E, D, seed=91, scale=0.3), gen(E, seed=92, scale=0.1)
    ids_w, wts_w, _ = P.moe_route(h.double(), wr.double(), b.double() if bias else None, k, norm, scaling)
    ids = torch.empty(M, k, dtype=torch.int32, device=DEV)
    wts = torch.empty(M, k, device=DEV)
    K().moe_router(ids, wts, h.to(DEV), wr.to(DEV), b.to(DEV) if bias else None, norm, scaling)
    assert torch.equal(ids.cpu().long(), ids_w)
    assert err(wts, wts_w) < 1e-5
    offs = torch.empty(E + 1, dtype=torch.int32, device=DEV)
    sp = torch.empty(M * k, dtype=torch.int32, device=DEV)
    pr = torch.empty(M * k, dtype=torch.int32, device=DEV)
    K().moe_align(offs, sp, pr, ids, E)
    flat = ids_w.reshape(-1)
    order = torch.sort(flat, stable=True).indices              # stable in the pair index
    assert torch.equal(sp.cpu().long(), order)
    assert torch.equal(offs.cpu().long(), torch.cat([torch.zeros(1, dtype=torch.long), torch.bincount(flat, minlength=E).cumsum(0)]))
    assert torch.equal(pr.cpu().long()[order], torch.arange(M * k))
    ys = gen(M * k, D, seed=93)
    x = gen(M, D, seed=94).to(DEV)
    x0 = x.cpu().double()
    K().moe_combine(x, ys.to(DEV), pr, wts, True)
    want = x0 + (wts_w[:, :, None] * ys.double()[pr.cpu().long().view(M, k)]).sum(1)
    assert err(x, want) < 1e-5


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("E,k,D", [(32, 4, 2048), (8, 2, 104), (5, 1, 72), (64, 6, 520), (10, 3, 4104), (9, 2, 768), (8, 1, 760), (23, 4, 536)])
def test_moe_router_gives_a_row_the_same_bits_whatever_the_step(dtype, E, k, D):
    """The router has a form of four blocks a row (up to 37 rows on 148 SMs; a quarter of the experts each, whole or not, and rows of
    more than one round of 2,048), one of a block a row and forms of several rows a block (many rows): a row's experts and
    weights are the same bits in all of them, so that a token is routed the same way alone, in a decode batch and
    inside a prompt."""
    M = 700
    h = gen(M, D, seed=97, dtype=dtype).to(DEV)
    wr, b = gen(E, D, seed=98, scale=0.3).to(DEV), gen(E, seed=99, scale=0.1).to(DEV)
    def route(rows, ahead=False):
        ids = torch.empty(rows.shape[0], k, dtype=torch.int32, device=DEV)
        wts = torch.empty(rows.shape[0], k, device=DEV)
        K().moe_router(ids, wts, rows, wr, b, True, 1.5, ahead=ahead)
        return ids, wts
    all_ids, all_w = route(h)                                  # many rows: four per block
    some_ids, some_w = route(h[:200].contiguous())
    assert torch.equal(some_ids, all_ids[:200]) and torch.equal(some_w, all_w[:200])
    last = K().sm_count() // 4                                 # rows up to which a row has four blocks
    for n in (1, 7, last, last + 1, 64, K().sm_count(), K().sm_count() + 1):
        for lo in (0, 199, M - n):
            for ahead in (False, True):
                ids, wts = route(h[lo:lo + n].contiguous(), ahead)
                assert torch.equal(ids, all_ids[lo:lo + n]) and torch.equal(wts, all_w[lo:lo + n])
    want_ids, want_w, _ = P.moe_route(h.double().cpu(), wr.double().cpu(), b.double().cpu(), k, True, 1.5)
    agree = (all_ids.cpu().long() == want_ids).all(dim=1)
    assert agree.float().mean() > 0.97                        # the rest: near-ties at float rounding
    assert err(all_w[agree.to(DEV)], want_w[agree]) < 1e-5


def test_moe_router_reads_weights_that_the_launch_before_it_wrote():
    """Unless the caller says otherwise (`ahead`), router rows may come from one of the library's own kernels launched right
    before: here a 32-bit product, which lets the router's blocks start at its beginning and writes at its end."""
    M, E, D, k, inner = 8, 32, 2048, 4, 4096
    h, x, w = gen(M, D, seed=30).to(DEV), gen(E, inner, seed=31, scale=inner ** -0.5).to(DEV), gen(D, inner, seed=32, scale=0.1).to(DEV)
    wr, ids, wts = torch.empty(E, D, device=DEV), torch.empty(M, k, dtype=torch.int32, device=DEV), torch.empty(M, k, device=DEV)
    def run():
        K().linear(wr, x, w)
        K().moe_router(ids, wts, h, wr, None, True, 1.0)
    run()
    K().linear(wr, x, w)
    torch.cuda.synchronize()
    K().moe_router(ids, wts, h, wr, None, True, 1.0)
    want = ids.clone(), wts.clone()
    graph = torch.cuda.CUDAGraph()      # the second launch right behind the first
    with torch.cuda.graph(graph):
        run()
    for _ in range(20):
        wr.zero_()
        torch.cuda.synchronize()
        graph.replay()
        assert torch.equal(ids, want[0]) and torch.equal(wts, want[1])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,k,E,D", [(1, 1, 1, 8), (1, 4, 32, 2048), (8, 4, 32, 2048), (64, 4, 32, 520), (51, 5, 256, 4100), (37, 2, 3, 72),
                                     (1, 1, 256, 64), (4, 8, 256, 2048), (33, 1, 256, 72), (11, 1, 32, 64), (3, 4, 32, 64),
                                     (65, 4, 32, 64), (9, 3, 8, 36)])
def test_moe_align_gather(dtype, M, k, E, D):
    """The expert-sorted order and the rows in it by one launch (up to 256 pairs, rows of whole 16-byte pieces; the last two
    sizes are beyond): what the sort and the gather give, with and without weights on the rows; fewer pairs than experts,
    experts without rows, more pieces than threads; offsets counted by a thread each (up to 32 pairs for 256 experts, 11 for 32)
    and by whole blocks."""
    g = torch.Generator().manual_seed(7 * M + k)
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(M)]).to(torch.int32).to(DEV)
    h, w = gen(M, D, seed=90, dtype=dtype).to(DEV), gen(M, k, seed=91).to(DEV)
    for weights in (None, w):
        want, got = [], []
        for out in (want, got):
            i32 = lambda n: torch.full((n,), -1, dtype=torch.int32, device=DEV)  # noqa: E731
            out += [i32(E + 1), i32(M * k), i32(M * k), torch.full((M * k, D), float("nan"), dtype=dtype, device=DEV)]
        K().moe_align(*want[:3], ids, E)
        K().gather_rows(want[3], h, want[1], div=k, weights=weights)
        K().moe_align_gather(*got, ids, h, E, weights=weights)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


# ---- sampling ---------------------------------------------------------------------------------------------
@pytest.mark.parametrize("V", [256, 1000, 65536])
def test_argmax_and_sampling(V):
    n = 6
    logits = gen(n, V, seed=95, scale=3.0)
    logits[2, 17] = logits[2, 400 % V] = logits[2].max() + 1       # a tie: the lower id wins
    if V >= 4096:
        # a row laid out against the kernel's quick way: the largest values all fall to the same few
        # threads (ids that are equal modulo 1024), so thousands of values reach the bound it takes
        # from the threads' maxima and it has to select over the whole row
        order = torch.argsort(logits[5], descending=True)
        ids = torch.arange(V)
        place = (ids % 1024) * (V // 1024) + ids // 1024            # rank of id i in that layout
        logits[5] = logits[5][order][place]
    ld = logits.to(DEV)
    out = torch.empty(n, dtype=torch.int32, device=DEV)
    K().argmax(out, ld)
    assert out.cpu().tolist() == [int(np.argmax(r)) for r in logits.numpy()]
    for temperature, top_k, top_p, min_p in ((0.8, 40, 0.95, 0.0), (1.3, 0, 1.0, 0.05), (0.5, 500, 0.5, 0.0), (1.0, 1, 0.0, 0.0)):
        for trial in range(4):
            u = np.random.default_rng(trial).random(n).astype(np.float32)
            K().sample(out, ld, torch.from_numpy(u).to(DEV), top_k, temperature, top_p, min_p)
            want = [P.sample(logits[i].numpy(), temperature, top_k, top_p, min_p, float(u[i])) for i in range(n)]
            assert out.cpu().tolist() == want, (temperature, top_k, top_p, min_p, trial)


def test_penalties():
    V = 50
    logits = gen(2, V, seed=96)
    hist = torch.zeros(2, 256, dtype=torch.int32)
    hist[0, :4] = torch.tensor([3, 7, 3, 9])
    ln = torch.tensor([4, 0], dtype=torch.int32)
    want = logits.clone()
    for t in [3, 7, 3, 9]:
        v = want[0, t]
        want[0, t] = (v / 1.3 if v > 0 else v * 1.3) - 0.2
    ld = logits.to(DEV)
    K().penalties(ld, hist.to(DEV), ln.to(DEV), 1.3, 0.2)
    assert err(ld, want) < 1e-6


# ---- the tcgen05 matrix product ------------------------------------------------------------------
@pytest.mark.parametrize("M,N,K_", [(128, 128, 64), (128, 256, 128), (65, 48, 72), (200, 100, 200), (300, 520, 136),
                                    (2048, 2048, 2048), (513, 6144, 2048), (1000, 2048, 5632),
                                    (17, 2048, 256), (64, 352, 128), (100, 6144, 64), (33, 11264, 192)])
def test_linear_tc(M, N, K_):
    """Tensor-memory accumulation against float64, at tile-aligned sizes and at sizes where rows,
    columns and k all run past the last tile; store, add-to-residual, and both result types."""
    x, w = gen(M, K_, seed=100, dtype=torch.bfloat16), gen(N, K_, seed=101, dtype=torch.bfloat16)
    want = x.double() @ w.double().T
    out = torch.full((M, N), float("nan"), device=DEV)
    assert K().linear_tc(out, x.to(DEV), w.to(DEV))
    K().check_device_status()
    assert err(out, want) < 2e-5
    ob = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    K().linear_tc(ob, x.to(DEV), w.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(M, N, seed=102).to(DEV)
    b0 = base.clone()
    K().linear_tc(base, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    K().check_device_status()
    assert err(base, b0.cpu().double() + want) < 2e-5


@pytest.mark.parametrize("M,N,K_", [(300, 2048, 4096), (512, 2048, 5632), (200, 3072, 8192), (130, 264, 6080), (257, 1000, 4104)])
def test_linear_tc_with_k_in_slices(M, N, K_):
    """Products of a few hundred rows with a long K (prompts of that length, the down projection):
    fewer 128 x 256 tiles than SMs, so K is cut into slices whose partial tiles a second kernel adds
    up.  Store, add to the residual and SwiGLU against float64; a last slice with fewer k-blocks,
    rows and columns past the tiles."""
    from lastengine_b200.parts.ffn import fuse_gate_up
    assert K().lib().leb_gemm_bf16_tc_slices(M, N, K_) > 1
    x, w = gen(M, K_, seed=110, dtype=torch.bfloat16), gen(N, K_, seed=111, scale=0.05, dtype=torch.bfloat16)
    want = x.double() @ w.double().T
    out = torch.full((M, N), float("nan"), device=DEV)
    assert K().linear_tc(out, x.to(DEV), w.to(DEV))
    assert err(out, want) < 2e-5
    ob = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    K().linear_tc(ob, x.to(DEV), w.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(M, N, seed=112).to(DEV)
    b0 = base.clone()
    K().linear_tc(base, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    assert err(base, b0.cpu().double() + want) < 2e-5
    again = b0.clone()
    K().linear_tc(again, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    assert torch.equal(again, base)                  # the slices are added in a fixed order
    if N % 32 == 0:
        F = N // 2
        o2 = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
        K().linear_tc(o2, x.to(DEV), fuse_gate_up(w[:F], w[F:], True).to(DEV), K().SWIGLU)
        assert err(o2, P.silu(want[:, :F]) * want[:, F:]) < 6e-3
    K().check_device_status()


@pytest.mark.parametrize("M,F,D", [(128, 64, 64), (70, 16, 40), (300, 160, 96), (2048, 5632, 2048), (40, 5632, 128), (64, 1024, 64)])
def test_linear_tc_swiglu_epilogue(M, F, D):
    from lastengine_b200.parts.ffn import fuse_gate_up
    x = gen(M, D, seed=103, dtype=torch.bfloat16)
    w1, w3 = gen(F, D, seed=104, scale=0.05, dtype=torch.bfloat16), gen(F, D, seed=105, scale=0.05, dtype=torch.bfloat16)
    want = P.silu(x.double() @ w1.double().T) * (x.double() @ w3.double().T)
    w13 = fuse_gate_up(w1, w3, True).to(DEV)
    out = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
    assert K().linear_tc(out, x.to(DEV), w13, K().SWIGLU)
    K().check_device_status()
    assert err(out, want) < 6e-3


def test_linear_tc_strided_operand_and_small_kernel_agree():
    """A column slice as the left operand (row stride larger than its width), and agreement with the
    weight-streaming kernel on the same product."""
    M, N, K_ = 150, 96, 128
    big = gen(M, 3 * K_, seed=106, dtype=torch.bfloat16).to(DEV)
    x = big[:, K_:2 * K_]
    w = gen(N, K_, seed=107, dtype=torch.bfloat16).to(DEV)
    a = torch.empty(M, N, device=DEV)
    b = torch.empty(M, N, device=DEV)
    assert K().linear_tc(a, x, w)
    K().lib().leb_gemm_bf16_small(b.data_ptr(), 0, x.data_ptr(), w.data_ptr(), M, N, K_, x.stride(0), N, 0, None, 1, 0, M,
                                  torch.cuda.current_stream().cuda_stream)
    assert err(a, x.double().cpu() @ w.double().cpu().T) < 2e-5
    assert err(a, b) < 2e-6


def test_shortconv_kernels_against_the_references_own():
    """The engine's convolution kernels (rows + state, and the one-launch decode form) on the inputs
    of tests/golden/shortconv_golden.npz, which holds what the reference's kernels gave."""
    import os
    g = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "shortconv_golden.npz"))
    for case in range(3):
        bcx, w = torch.from_numpy(g[f"bcx{case}"]), torch.from_numpy(g[f"w{case}"])
        T, n, lc = bcx.shape[0], w.shape[0], w.shape[1]
        for mode in ("chunk", "steps"):
            state = torch.zeros(3, n, lc - 1, device=DEV)
            state[2] = torch.from_numpy(g[f"state_in{case}"]).to(DEV)
            y = torch.empty(T, n, device=DEV)
            bb = builder()
            if mode == "chunk":
                K().shortconv(y, bcx.to(DEV), w.to(DEV), None, state, bb.build([2], [[0] * T], [0], [], {}), lc)
            else:
                for t in range(T):
                    K().shortconv(y[t:t + 1], bcx[t:t + 1].to(DEV), w.to(DEV), None, state, bb.build([2], [[0]], [t], [], {}), lc)
            assert err(y, torch.from_numpy(g[f"y{case}"])) < 1e-6, (case, mode)
            assert err(state[2], torch.from_numpy(g[f"state_out{case}"])) < 1e-6, (case, mode)


@pytest.mark.parametrize("M,N,K_", [(256, 256, 64), (300, 520, 136), (129, 100, 72), (1000, 2048, 5632), (2048, 6144, 2048),
                                    (2700, 1544, 136), (4100, 520, 328)])
def test_linear_tc_pairs(M, N, K_):
    """The product on pairs of SMs (cta_group::2, 256 x 256 tiles): tile-aligned sizes and sizes where
    rows, columns and k run past the last tile, a last band of fewer row tiles than eight behind whole ones among them; store, add to the residual, SwiGLU, both result types."""
    x, w = gen(M, K_, seed=100, dtype=torch.bfloat16), gen(N, K_, seed=101, scale=0.05, dtype=torch.bfloat16)
    want = x.double() @ w.double().T
    out = torch.full((M, N), float("nan"), device=DEV)
    assert K().linear_tc2(out, x.to(DEV), w.to(DEV))
    K().check_device_status()
    assert err(out, want) < 2e-5
    ob = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    K().linear_tc2(ob, x.to(DEV), w.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(M, N, seed=102).to(DEV)
    b0 = base.clone()
    K().linear_tc2(base, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    assert err(base, b0.cpu().double() + want) < 2e-5
    if N % 32 == 0:
        from lastengine_b200.parts.ffn import fuse_gate_up
        F = N // 2
        w13 = fuse_gate_up(w[:F], w[F:], True).to(DEV)
        o2 = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
        K().linear_tc2(o2, x.to(DEV), w13, K().SWIGLU)
        assert err(o2, P.silu(want[:, :F]) * want[:, F:]) < 6e-3
    K().check_device_status()


@pytest.mark.parametrize("M,N,K_", [(6144, 2040, 264), (16200, 300, 1032), (32767, 257, 1024), (16200, 300, 1016), (4000, 2056, 1032)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_linear_of_many_tiles_of_a_narrow_matrix(M, N, K_, dtype):
    """Matrices of less than 4,096 either way on both sides of the line from which their products run on pairs of SMs, with part
    tiles of rows, columns and k.  Sums of K_ bfloat16 products in float; a bfloat16 result is rounded once more."""
    x, w = gen(M, K_, seed=120, dtype=torch.bfloat16).to(DEV), gen(N, K_, seed=121, scale=0.05, dtype=torch.bfloat16).to(DEV)
    out = torch.full((M, N), float("nan"), device=DEV, dtype=dtype)
    K().linear(out, x, w)
    K().check_device_status()
    want = (x.double() @ w.double().T).cpu()
    assert err(out, want) < (2e-5 if dtype == torch.float32 else 5e-3)
    if dtype == torch.float32:
        base = gen(M, N, seed=122).to(DEV)
        b0 = base.clone()
        K().linear(base, x, w, K().ACCUMULATE)
        assert err(base, b0.cpu().double() + want) < 2e-5


@pytest.mark.parametrize("M,N,K_", [(17, 2048, 2048), (64, 352, 128), (100, 6144, 64), (33, 11264, 192), (128, 100, 200),
                                    (1, 128, 64), (16, 48, 72), (48, 2048, 5632), (64, 65536, 256),
                                    (65, 2048, 2048), (96, 352, 5632), (90, 100, 200), (97, 6144, 136),
                                    (24, 100, 1024), (24, 100, 1280), (24, 100, 2048), (24, 100, 2304), (24, 100, 4096), (24, 100, 4352), (40, 100, 8192)])
def test_linear_skinny(M, N, K_):
    """The swapped-operand tcgen05 product with K sliced over blocks: store, add to residual, both
    result types, sizes that leave partial tiles and slices; 4 and 5, 8 and 9, 16 and 17, and 32 slices (the second
    kernel asks for up to 4, 8 or 16 at a time)."""
    x, w = gen(M, K_, seed=120, dtype=torch.bfloat16), gen(N, K_, seed=121, scale=0.05, dtype=torch.bfloat16)
    want = x.double() @ w.double().T
    out = torch.full((M, N), float("nan"), device=DEV)
    assert K().linear_skinny(out, x.to(DEV), w.to(DEV))
    K().check_device_status()
    assert err(out, want) < 2e-5
    ob = torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
    K().linear_skinny(ob, x.to(DEV), w.to(DEV))
    assert err(ob, want) < 5e-3
    base = gen(M, N, seed=122).to(DEV)
    b0 = base.clone()
    K().linear_skinny(base, x.to(DEV), w.to(DEV), K().ACCUMULATE)
    K().check_device_status()
    assert err(base, b0.cpu().double() + want) < 2e-5


@pytest.mark.parametrize("M,F,D", [(64, 5632, 2048), (20, 16, 40), (100, 160, 96), (80, 5632, 2048), (96, 160, 96)])
def test_linear_skinny_swiglu(M, F, D):
    from lastengine_b200.parts.ffn import fuse_gate_up
    x = gen(M, D, seed=123, dtype=torch.bfloat16)
    w1, w3 = gen(F, D, seed=124, scale=0.05, dtype=torch.bfloat16), gen(F, D, seed=125, scale=0.05, dtype=torch.bfloat16)
    want = P.silu(x.double() @ w1.double().T) * (x.double() @ w3.double().T)
    out = torch.empty(M, F, device=DEV, dtype=torch.bfloat16)
    assert K().linear_skinny(out, x.to(DEV), fuse_gate_up(w1, w3, True).to(DEV), K().SWIGLU)
    K().check_device_status()
    assert err(out, want) < 6e-3


def _gate(name, g, u):
    if name == "silu":
        return P.silu(g) * u
    if name == "gelu_tanh":
        return 0.5 * g * (1 + torch.tanh(math.sqrt(2 / math.pi) * (g + 0.044715 * g ** 3))) * u
    g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
    return g * torch.sigmoid(1.702 * g) * (u + 1)


@pytest.mark.parametrize("M,D,F,gate", [(17, 64, 16, "silu"), (32, 2048, 5632, "silu"), (33, 104, 176, "gelu_tanh"), (64, 2048, 7168, "silu"),
                                        (48, 520, 1040, "clamped"), (65, 1000, 2000, "silu"), (96, 328, 4224, "gelu_tanh"),
                                        (97, 264, 96, "clamped"), (128, 2048, 1536, "silu")])
def test_product_chain(M, D, F, gate):
    """Products of a step run as one resident kernel: convolution, sum with the next norm's half, gated epilogue, store with and
    without an activation, float and bfloat16, twice over (a second layer reads what the first wrote); rows at the edges of
    the paddings, K of one block and of part blocks, tiles of every height, padding sequences.  Each product against
    64 bits from the inputs it had; a product that adds up to K terms of bfloat16 in float is off by at most 2e-5 of the largest,
    a bfloat16 result by half a step more (8 significant bits: at most 2^-8 of the value), the convolution by that of its three
    projections and of its own."""
    import types
    from lastengine_b200.engine.workspace import Workspace
    from lastengine_b200.parts.ffn import fuse_gate_up
    k = K()
    ws, b16, f32 = Workspace(torch.device(DEV)), torch.bfloat16, torch.float32
    if k.lib().leb_gemm_bf16_skinny_slices(3 * D, D) < 2:
        conv_fits = False        # the convolution alone needs two slices: the chain then begins without it
    else:
        conv_fits = True
    slot = torch.arange(M, dtype=torch.int32).flip(0)
    slot[M // 2] = -1
    batch = types.SimpleNamespace(max_qlen=1, n_seqs=M, row_seq=torch.arange(M, dtype=torch.int32, device=DEV), seq_slot=slot.to(DEV))
    act = {"silu": k.SILU, "gelu_tanh": k.GELU_TANH, "clamped": k.CLAMPED_SIGMOID}[gate]
    gated = k.gated_epilogue(act, 7.0 if gate == "clamped" else 0.0, 1.702 if gate == "clamped" else 1.0)
    W = {n: gen(r, c, seed=i, scale=c ** -0.5, dtype=b16) for i, (n, (r, c)) in enumerate(
        {"in": (3 * D, D), "o": (D, D), "g": (F, D), "u": (F, D), "down": (D, F), "head": (F, D)}.items())}
    taps, bias, norm = gen(D, 3, seed=20), gen(D, seed=21, scale=0.1), 1 + gen(D, seed=22, scale=0.1)
    dev = {n: t.to(DEV) for n, t in W.items()}
    dev["gu"] = fuse_gate_up(W["g"], W["u"], True).to(DEV)
    h, x0, st0 = gen(M, D, seed=23, dtype=b16), gen(M, D, seed=24), gen(M, D, 2, seed=25)
    x, st, hd = x0.to(DEV), st0.to(DEV), torch.zeros(M, D + 16, dtype=b16, device=DEV)[:, :D]     # rows of a wider matrix
    hd.copy_(h)
    buf = lambda *shape, dtype=b16: torch.full(shape, float("nan"), dtype=dtype, device=DEV)  # noqa: E731
    steps, inp, scale = [], hd, None
    before = k.launch_count()
    with k.product_chain(ws, M, b16):
        for layer in range(2):
            y = buf(M, D)
            if conv_fits:
                assert k.shortconv_decode_fused(y, inp, dev["in"], taps.to(DEV), bias.to(DEV), st, batch, 3, scale=scale)
            else:
                k.linear(y, inp, dev["o"], scale=scale)
            mid = k.SplitNorm(buf(M, D), buf(M, -(-D // 16), dtype=f32), norm.to(DEV), 1e-5)
            k.linear(x, y, dev["o"], k.ACCUMULATE, emit=mid)
            a = buf(M, F)
            k.linear(a, mid.values, dev["gu"], gated, scale=mid)
            nxt = k.SplitNorm(buf(M, D), buf(M, -(-D // 16), dtype=f32), norm.to(DEV), 1e-5)
            k.linear(x, a, dev["down"], k.ACCUMULATE, emit=nxt)
            steps.append((inp, scale, y, mid, a, nxt))
            inp, scale = nxt.values, nxt
        z, zf = buf(M, F + 24)[:, 8:8 + F], buf(M, F + 3, dtype=f32)[:, 3:]
        k.linear(z, inp, dev["head"], k.plain_act_epilogue(k.PLAIN_ACTIVATIONS["relu_squared"]), scale=scale)
        k.linear(zf, inp, dev["head"], scale=scale)
    k.check_device_status()
    assert k.launch_count() - before == 1
    assert ws.zeroed("chain.sync", 2).tolist() == [0, 0]

    def rows(values, sc):      # the rows a product read: with a split norm, values times the rows' factor
        v = values.double().cpu()
        return v if sc is None else v / torch.sqrt(sc.ssq.double().cpu().sum(-1, keepdim=True) / D + 1e-5)
    want_x, state = x0.double(), st0.double()
    for inp, sc, y, mid, a, nxt in steps:
        v = rows(inp, sc)
        if conv_fits:
            b, c, u = (v @ W["in"].double().T).chunk(3, -1)
            on = slot >= 0
            bx = b.to(b16).double() * u.to(b16).double()
            old = state[slot.clamp(min=0).long()]
            conv = old[:, :, 0] * taps[:, 0].double() + old[:, :, 1] * taps[:, 1].double() + bx * taps[:, 2].double() + bias.double()
            want = torch.where(on[:, None], c.to(b16).double() * conv, torch.zeros(()).double())
            state = state.clone()
            state[slot[on].long()] = torch.stack([old[:, :, 1], bx], -1)[on]
            assert err(y, want) < 4 * 2 ** -8
        else:
            assert err(y, v @ W["o"].double().T) < 2 ** -8 + 2e-5
        want_x = want_x + y.double().cpu() @ W["o"].double().T
        assert err(mid.values, want_x * norm.double()) < 2 ** -8 + 2e-5
        v = rows(mid.values, mid)
        assert err(a, _gate(gate, v @ W["g"].double().T, v @ W["u"].double().T)) < 2 ** -8 + 1e-4
        want_x = want_x + a.double().cpu() @ W["down"].double().T
        assert err(nxt.values, want_x * norm.double()) < 2 ** -8 + 2e-5
        assert err(nxt.ssq.sum(-1), (want_x ** 2).sum(-1)) < 1e-4
    assert err(x, want_x) < 2e-5
    if conv_fits:
        assert err(st, state) < 2 * 2 ** -8
    v = rows(steps[-1][5].values, steps[-1][5]) @ W["head"].double().T
    assert err(zf, v) < 2e-5 and err(z, torch.clamp(v, min=0) ** 2) < 2 ** -8 + 4e-5

