"""Products that wait for one another on the host: nothing but the library's own code runs while they wait.

The models run here without a GPU: the kernel library is replaced by one that computes nothing and counts what waits."""
import dataclasses
import weakref

import pytest
import torch

import kisilix_configs
import lenesun_configs
import nolapel_configs
import tevilix_configs
import tiny_configs
import zafilix_configs
import zekivik_configs
from lastengine_b200 import registry
from lastengine_b200.cache.cache import Cache, pooled_table_key
from lastengine_b200.engine.batch import BatchBuilder
from lastengine_b200.engine.model import Model
from lastengine_b200.engine.workspace import Workspace
from lastengine_b200.ops import kernels
from lastengine_b200.parts.base import BuildEnv

CONFIGS = {f"{mod.__name__.removesuffix('_configs')}_{name}": cfg for mod in (tiny_configs, zekivik_configs, lenesun_configs, kisilix_configs, tevilix_configs, zafilix_configs,
                                 nolapel_configs)
           for name, cfg in vars(mod).items() if isinstance(cfg, dict) and ("architecture" in cfg or "architectures" in cfg)}
# what a forward pass calls of a part
ENTRIES = ("forward", "forward_parts", "apply", "fused_rotary", "add_gated", "add_into", "give_rows_to")
ROWS = 20
CPU = torch.device("cpu")


class CountingLibrary:
    """Every entry point does nothing and answers 0; the products and the launches of chains are counted."""

    def __init__(self):
        self.waiting = self.chains = self.dropped = 0      # waiting: added, not launched
        self.longest = 0

    def leb_chain_clusters(self, rows):
        return 33

    def leb_chain_max_ops(self):
        return 40

    def leb_chain_takes(self, m, n, k):
        return 1

    def leb_gemm_bf16_skinny_slices(self, n, k):
        return 4

    def leb_sm_count(self):
        return 148

    def leb_chain_add(self, *a):
        self.waiting += 1
        self.longest = max(self.longest, self.waiting)
        return 0

    def leb_chain_run(self, *a):
        self.waiting, self.chains = 0, self.chains + 1
        return 0

    def leb_chain_drop(self):
        self.waiting, self.dropped = 0, self.dropped + 1
        return 0

    def leb_last_error(self):
        return b"refused"

    def __getattr__(self, name):
        if name.startswith("leb_"):
            return lambda *a: 0
        raise AttributeError(name)


@pytest.fixture
def library(monkeypatch):
    lib = CountingLibrary()
    monkeypatch.setattr(kernels, "_lib", lib)
    monkeypatch.setattr(kernels, "_timer", None)
    monkeypatch.setattr(kernels, "_cuda", lambda *a, **k: None)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    monkeypatch.setattr(kernels, "_tc_block", {})
    monkeypatch.setattr(kernels, "_device_index", lambda d: 0)
    monkeypatch.setattr(kernels, "sm_count", lambda: 148)
    monkeypatch.setattr(kernels, "chain_pays", lambda rows, sizes: len(sizes) >= 2)
    monkeypatch.setattr(kernels, "_tc_status", {})
    monkeypatch.setattr(kernels, "_retention_ws", {})
    monkeypatch.setattr(kernels, "_gru_piece", [64])
    monkeypatch.setattr(kernels, "_skinny_workspace", lambda d, n: torch.empty(n))
    yield lib
    assert not kernels._chain.open and not kernels._chain.ops and lib.waiting == 0


def make(plan) -> Model:
    env = BuildEnv(device=CPU, dtype=torch.bfloat16, workspace=Workspace(CPU))
    m = Model(plan, env)
    g = torch.Generator().manual_seed(1)
    m.load({n: torch.randn(s.concrete_shape(), generator=g).to(torch.bfloat16 if s.role in ("matrix", "embedding") else torch.float32)
            for n, s in m.tensor_specs().items()})
    return m


def forward(m: Model, rows=ROWS, seqs=1):
    """A step of `rows` rows, the prompts of `seqs` new sequences of equal lengths."""
    cache = Cache(m.cache_specs(), max_tokens=128 * (seqs + 2), max_seqs=seqs + 1, dtype=torch.bfloat16, device=CPU)
    slots = [cache.alloc_seq() for _ in range(seqs)]
    cache.reserve({s: rows // seqs for s in slots})
    tables = {}
    for gi, g in enumerate(cache.kv_groups):
        tables[gi] = g.table(slots, 2)
        if g.pool > 0:
            tables[pooled_table_key(gi)] = g.table(slots, 2, pooled=True)
    batch = BatchBuilder(CPU).build(slots, [[1] * (rows // seqs)] * seqs, [0] * seqs, [rows - 1], tables)
    return m.forward(batch, cache)


def parts_of(m: Model) -> list:
    return [p for p in m._objects_in([*m.blocks, m.embedding, m.final_norm, m.head], {}) if any(hasattr(p, n) for n in ENTRIES)]


def spied(method, library, seen: list):
    """`method` as other code would wrap it: notes what waits when it begins and when it ends."""
    def spy(*a, **k):
        seen.append((kernels._chain.open, len(kernels._chain.ops), library.waiting))
        out = method(*a, **k)
        seen.append((kernels._chain.open, len(kernels._chain.ops), library.waiting))
        return out
    return spy


@pytest.mark.parametrize("name", sorted(CONFIGS))
def test_a_wrapped_part_finds_nothing_waiting(name, library):
    """Every part of every design, wrapped on a built model in turn: when its method runs, whatever waited has been launched,
    and its own products do not wait.  The model without wraps is the library's own."""
    m = make(registry.plan_from_config(CONFIGS[name]))
    assert m.chains
    called = 0
    for part in parts_of(m):
        seen: list = []
        names = [n for n in ENTRIES if hasattr(part, n)]
        for n in names:
            setattr(part, n, spied(getattr(part, n), library, seen))
        for seqs in (1, ROWS):
            forward(m, seqs=seqs)
        for n in names:
            delattr(part, n)
        assert all(s == (False, 0, 0) for s in seen), (type(part).__name__, seen)
        called += bool(seen)
    assert called >= 2 * len(m.blocks)


@pytest.mark.parametrize("way", ["subclass", "class"])
@pytest.mark.parametrize("name", ["tiny_TINY_A", "tiny_TINY_C", "zekivik_Z_A", "zekivik_Z_B"])
def test_a_part_of_another_class_finds_nothing_waiting(name, way, library, monkeypatch):
    """The same for a part replaced by one of a class from elsewhere, and for a method replaced on the library's class."""
    m = make(registry.plan_from_config(CONFIGS[name]))
    for part in parts_of(m):
        seen: list = []
        own = type(part)
        with monkeypatch.context() as patch:
            if way == "subclass":
                part.__class__ = type("Elsewhere", (own,), {"__module__": __name__})
            for n in [n for n in ENTRIES if hasattr(part, n)]:
                patch.setattr(type(part), n, spied(getattr(own, n), library, seen), raising=False)
            for seqs in (1, ROWS):
                forward(m, seqs=seqs)
        part.__class__ = own
        assert all(s == (False, 0, 0) for s in seen), (own.__name__, seen)


def test_products_wait_between_parts_of_the_library(library):
    """What the tests above rely on: without other code, products of several parts wait together."""
    m = make(registry.plan_from_config(CONFIGS["tiny_TINY_A"]))
    forward(m, seqs=ROWS)
    assert library.chains >= 2 and library.longest >= 4
    whole = library.longest
    m.blocks[1].ffn.forward = spied(m.blocks[1].ffn.forward, library, [])
    library.chains = library.longest = 0
    forward(m, seqs=ROWS)
    assert library.chains >= 1 and 2 <= library.longest < whole


ROLES = {"mixer": registry.MIXERS, "ffn": registry.FEED_FORWARDS, "mixer_norm": registry.NORMS, "ffn_norm": registry.NORMS,
         "gate": registry.GATES, "position": registry.POSITION_ENCODINGS, "block": registry.BLOCKS,
         "embedding": registry.EMBEDDINGS, "head": registry.HEADS, "final_norm": registry.NORMS}


@pytest.mark.parametrize("role", list(ROLES))
def test_a_model_built_with_a_part_from_elsewhere_launches_every_product_at_once(role, library):
    """A registered class of every kind, gates and position encodings (which have no `forward`) among them."""
    plan = registry.plan_from_config(CONFIGS["zekivik_Z_A"])
    at = next(i for i, ls in enumerate(plan.layers) if ls.gates and ls.ffn is not None)
    ls = plan.layers[at]
    if role == "gate":
        name, spec = next(iter(ls.gates.items()))
    elif role == "position":
        spec = ls.mixer.params["position"]
    else:
        spec = getattr(ls, role, None) or getattr(plan, role)
    kind = spec if role == "block" else spec.kind
    elsewhere = type("Elsewhere", (ROLES[role].get(kind),), {"__module__": __name__})
    ROLES[role].register("from_elsewhere")(elsewhere)
    try:
        new = "from_elsewhere" if role == "block" else dataclasses.replace(spec, kind="from_elsewhere")
        if role == "gate":
            ls = dataclasses.replace(ls, gates={**ls.gates, name: new})
        elif role == "position":
            mixer = dataclasses.replace(ls.mixer, params={**ls.mixer.params, "position": new})
            ls = dataclasses.replace(ls, mixer=mixer)
        elif hasattr(ls, role):
            ls = dataclasses.replace(ls, **{role: new})
        layers = [*plan.layers[:at], ls, *plan.layers[at + 1:]]
        changed = {role: new} if role in ("embedding", "head", "final_norm") else {}
        m = make(dataclasses.replace(plan, layers=layers, **changed))
        assert not m.chains
        forward(m)
        assert library.chains == library.longest == 0
    finally:
        ROLES[role].unregister("from_elsewhere")


def test_a_model_inside_a_part_has_a_chain_of_its_own(library):
    """A part from elsewhere that runs another model of the same rows reads its result: nothing of it waits any more, and the
    outer step goes on with its own barrier's words."""
    outer, inner = (make(registry.plan_from_config(CONFIGS["tiny_TINY_A"])) for _ in range(2))
    own, at = outer.blocks[1].ffn.forward, []

    def both(*a, **k):
        forward(inner)
        at.append((library.waiting, kernels._chain.open))
        return own(*a, **k)
    outer.blocks[1].ffn.forward = both
    after = outer.blocks[2].forward

    def noted(*a, **k):
        at.append(kernels._chain.sync)
        return after(*a, **k)
    outer.blocks[2].forward = noted
    forward(outer, seqs=ROWS)
    assert at[0] == (0, False) and at[1] is outer.env.workspace.zeroed("chain.sync", 2)


def test_a_part_that_raises_leaves_no_chain_behind(library):
    m = make(registry.plan_from_config(CONFIGS["tiny_TINY_A"]))

    def broken(*a, **k):
        raise ValueError("broken")
    m.blocks[2].ffn.forward = broken
    with pytest.raises(ValueError, match="broken"):
        forward(m, seqs=ROWS)
    del m.blocks[2].ffn.forward
    forward(m, seqs=ROWS)
    assert library.chains >= 2


@pytest.mark.parametrize("rows,products,uncut,mb,pays", [
    (17, 1, 0, 500, 0), (17, 1, 1, 500, 0), (17, 2, 1, 1, 1), (128, 2, 1, 1, 1), (17, 2, 0, 500, 0), (32, 2, 0, 500, 0), (32, 3, 0, 500, 0),
    (32, 4, 0, 1, 1), (24, 4, 0, 1, 1), (23, 4, 0, 500, 0), (17, 5, 0, 1, 1), (33, 2, 0, 500, 0), (33, 3, 0, 59, 0),
    (33, 3, 0, 61, 1), (48, 2, 0, 500, 0), (49, 2, 0, 1, 1), (64, 2, 0, 1, 1), (65, 2, 0, 500, 0), (65, 4, 0, 1, 1), (81, 2, 0, 1, 1),
    (97, 2, 0, 1, 1), (128, 2, 0, 1, 1)])
def test_which_products_run_as_a_chain(rows, products, uncut, mb, pays, monkeypatch):
    """The edges of the rule: rows, products, weights, and products whose K is not cut alone."""
    lib = CountingLibrary()
    lib.leb_gemm_bf16_skinny_slices = lambda n, k: 1 if uncut else 4
    monkeypatch.setattr(kernels, "_lib", lib)
    assert kernels.chain_pays(rows, [(mb * 500_000 // products, 1)] * products) == bool(pays)


def test_products_that_do_not_pay_as_a_chain_run_alone_in_their_order(library, monkeypatch):
    ran = []
    monkeypatch.setattr(kernels, "chain_pays", lambda rows, sizes: False)
    monkeypatch.setattr(library, "leb_gemm_bf16_skinny", lambda *a: ran.append(a[5]) or 0, raising=False)
    x, ws = torch.zeros(ROWS, 64, dtype=torch.bfloat16), Workspace(CPU)
    with kernels.product_chain(ws, ROWS, torch.bfloat16):
        for n in (32, 64, 96):
            kernels.linear(torch.zeros(ROWS, n), x, torch.zeros(n, 64, dtype=torch.bfloat16))
        assert len(kernels._chain.ops) == 3 and not ran
    assert ran == [32, 64, 96] and library.chains == library.longest == 0


def test_what_waits_keeps_its_operands(library):
    """A caller may let go of them: the launch comes later and takes addresses."""
    D, b16 = 64, torch.bfloat16
    ws, gone = Workspace(CPU), []

    def held(t):
        gone.append(weakref.ref(t))
        return t

    def add():
        sp = kernels.SplitNorm(held(torch.zeros(ROWS, D, dtype=b16)), held(torch.zeros(ROWS, 4)), held(torch.zeros(D)), 1e-5)
        x, w = held(torch.zeros(ROWS, D, dtype=b16)), held(torch.zeros(D, D, dtype=b16))
        kernels.linear(held(torch.zeros(ROWS, D)), x, w, kernels.ACCUMULATE, emit=sp)
        kernels.linear(held(torch.zeros(ROWS, D)), sp.values, w, scale=sp)
    with kernels.product_chain(ws, ROWS, b16):
        add()
        assert all(r() is not None for r in gone)
    assert library.chains == 1 and all(r() is None for r in gone)


def test_a_product_the_chain_refuses_when_it_is_launched_leaves_none_behind(library, monkeypatch):
    monkeypatch.setattr(library, "leb_chain_add", lambda *a: int(a[5] == 96), raising=False)
    x, ws = torch.zeros(ROWS, 64, dtype=torch.bfloat16), Workspace(CPU)
    with pytest.raises(kernels.KernelError, match="refused"), kernels.product_chain(ws, ROWS, torch.bfloat16):
        for n in (32, 96):
            kernels.linear(torch.zeros(ROWS, n), x, torch.zeros(n, 64, dtype=torch.bfloat16))
    assert library.chains == 0 and library.dropped == 1
