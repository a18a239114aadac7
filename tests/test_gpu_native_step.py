"""tx.step through the compiled plan (csrc/fo_host.cc) against the general path, bit for bit: trees of every container, each
optimizer, donated and not; and what must make a plan give way (edited param groups, selectors that change their mind,
gradients that need a conversion, several threads)."""

import collections
import contextlib
import threading

import pytest

pytestmark = pytest.mark.gpu

Pair = collections.namedtuple("Pair", "kernel bias")


def _params(seed=0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(s, device="cuda", generator=g) * 0.02
    return {"b": [Pair(r(33, 7).bfloat16(), r(7)), None], "a": {"w": r(70, 64).to(torch.float16), "z": (r(5).bfloat16(), r(2048).bfloat16())}}


def _grads(params, seed):
    import torch

    from flashoptim_jax_b200 import tree

    g = torch.Generator(device="cuda").manual_seed(seed)
    return tree.tree_map(lambda p: (torch.randn(p.shape, device="cuda", generator=g) * 1e-2).to(p.dtype), params)


def _leaves(x):
    from flashoptim_jax_b200 import tree

    return tree.tree_leaves(x)


def _same(a, b):
    import torch

    la, lb = _leaves(a), _leaves(b)
    assert len(la) == len(lb)
    for x, y in zip(la, lb):
        assert x.dtype == y.dtype and x.shape == y.shape and torch.equal(x.view(torch.uint8) if x.dim() else x, y.view(torch.uint8) if y.dim() else y)


@contextlib.contextmanager
def _general_path():
    from flashoptim_jax_b200 import _engine as eng

    eng.set_launch_observer(lambda key, n: contextlib.nullcontext())
    try:
        yield
    finally:
        eng.set_launch_observer(None)


FACTORIES = [("flash_adamw", dict(learning_rate=1e-3)), ("flash_adam", dict(learning_rate=lambda c: 1e-3 / (1 + int(c)), master_weight_bits=32, group_size=64)),
             ("flash_adamw", dict(learning_rate=1e-3, fused=False, quantize=False)), ("flash_lion", dict(weight_decay=1e-2)),
             ("flash_sgd", dict(learning_rate=1e-2)), ("flash_sgdw", dict(learning_rate=1e-2, momentum=0.9, nesterov=True, group_size=40, fused=False))]


@pytest.mark.parametrize("donate", [False, True])
@pytest.mark.parametrize("name,kw", FACTORIES)
def test_planned_steps_equal_general_steps(name, kw, donate, monkeypatch):
    import flashoptim_jax_b200 as fo

    groups = [{"params": ["bias", "a/z/1"], "weight_decay": 0.0, "learning_rate": 5e-3}, {"params": lambda p, leaf: leaf.dim() == 1, "weight_decay": 0.1}]
    tx = getattr(fo, name)(param_groups=groups, donate=donate, **kw)
    ref = getattr(fo, name)(param_groups=groups, **kw)
    p, q = _params(), _params()
    s, t = tx.init(p), ref.init(q)
    for k in range(4):
        g = _grads(q, k)
        before = [x.clone() for x in _leaves((p, s))]
        old = (p, s)
        with _only_planned_steps(monkeypatch) if k else contextlib.nullcontext():
            p, s = tx.step(p, s, g)
        with _general_path():
            q, t = ref.step(q, t, g)
        _same((p, tuple(s)), (q, tuple(t)))
        assert type(p["b"]) is list and type(p["b"][0]) is Pair and p["b"][1] is None and int(s.count) == k + 1
        if not donate:
            _same(old, before)


@pytest.mark.parametrize("donate", [False, True])
def test_edited_groups_and_selectors_are_honoured(donate):
    import torch

    import flashoptim_jax_b200 as fo

    frozen = set()
    groups = [{"params": lambda path, leaf: path[0] in frozen, "learning_rate": 0.0, "weight_decay": 0.0}, {"params": "y", "learning_rate": 2e-2}]
    tx = fo.flash_adamw(learning_rate=1e-2, param_groups=groups, donate=donate)
    p = {k: torch.ones(100, device="cuda", dtype=torch.bfloat16) for k in ("x", "y")}
    s, g = tx.init(p), {k: torch.full((100,), 0.1, device="cuda", dtype=torch.bfloat16) for k in ("x", "y")}
    for _ in range(3):
        p, s = tx.step(p, s, g)
    frozen.add("x")
    p0 = {k: v.clone() for k, v in p.items()}
    q, s = tx.step(p, s, g)
    assert torch.equal(q["x"], p0["x"]) and not torch.equal(q["y"], p0["y"])
    q0 = {k: v.clone() for k, v in q.items()}
    groups[1]["learning_rate"] = 0.0
    groups[1]["weight_decay"] = 0.0
    r, s = tx.step(q, s, g)
    assert torch.equal(r["y"], q0["y"])
    frozen.clear()
    r0 = r["x"].clone()
    r2, s = tx.step(r, s, g)
    assert not torch.equal(r2["x"], r0) and int(s.count) == 6


def test_selectors_are_asked_at_every_step():
    """Donated or not, the very same tensors or new ones: what a selector answers may depend on more than the leaf."""
    import torch

    import flashoptim_jax_b200 as fo

    asked = []
    tx = fo.flash_sgd(learning_rate=1e-2, donate=True, param_groups=[{"params": lambda path, leaf: asked.append(path) or False, "weight_decay": 0.0}])
    p = {"w": torch.ones(64, device="cuda", dtype=torch.bfloat16)}
    s, g = tx.init(p), {"w": torch.ones(64, device="cuda", dtype=torch.bfloat16)}
    for _ in range(3):
        p, s = tx.step(p, s, g)
    asked.clear()
    p, s = tx.step(p, s, g)
    assert asked == [("w",)]
    for _ in range(8):
        host = p["w"].cpu()
        del p["w"]  # the next tensor may get its address
        p["w"] = host.cuda()
        asked.clear()
        p, s = tx.step(p, s, g)
        assert asked


@pytest.mark.parametrize("donate", [False, True])
def test_a_call_without_elements_in_front(donate, monkeypatch):
    """The launch table that comes first holds only leaves without elements; the clipped launches behind it still wait for the norm."""
    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import clipping

    params = lambda: {"a": torch.ones(0, 3, device="cuda", dtype=torch.float16), "b": torch.ones(1 << 21, device="cuda"), "c": torch.ones(77, device="cuda", dtype=torch.bfloat16)}
    tx = clipping.clip_by_global_norm(fo.flash_adamw(learning_rate=1e-2, donate=donate), 1.0)
    ref = clipping.clip_by_global_norm(fo.flash_adamw(learning_rate=1e-2), 1.0)
    p, q = params(), params()
    s, t = tx.init(p), ref.init(q)
    for k in range(4):
        g = _grads(q, k)
        with _only_planned_steps(monkeypatch) if k else contextlib.nullcontext():
            p, s = tx.step(p, s, g)
        with _general_path():
            q, t = ref.step(q, t, g)
        _same((p, tuple(s["opt"])), (q, tuple(t["opt"])))


def test_gradients_that_need_a_conversion():
    import torch

    import flashoptim_jax_b200 as fo

    tx, ref = fo.flash_lion(donate=True), fo.flash_lion()
    p, q = {"w": torch.ones(64, 32, device="cuda", dtype=torch.bfloat16)}, {"w": torch.ones(64, 32, device="cuda", dtype=torch.bfloat16)}
    s, t = tx.init(p), ref.init(q)
    base = torch.randn(32, 64, device="cuda").bfloat16()
    for g in (base.t().contiguous(), base.t(), base.t().double(), base.t().float(), base.t().contiguous()):
        p, s = tx.step(p, s, {"w": g})
        with _general_path():
            q, t = ref.step(q, t, {"w": g.contiguous()})
        _same((p, s.mu, s.ecc), (q, t.mu, t.ecc))
    with pytest.raises(ValueError):
        tx.step(p, s, {"v": base})


def test_threads_share_an_optimizer():
    import time

    import torch

    import flashoptim_jax_b200 as fo

    def schedule(count):
        time.sleep(0.001)  # another thread steps meanwhile
        return 1e-3

    tx, ref = fo.flash_adamw(learning_rate=schedule, donate=True), fo.flash_adamw(learning_rate=1e-3)
    results, errors = {}, []

    def work(k):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                p = {"w": torch.full((3000,), 1.0 + k, device="cuda", dtype=torch.bfloat16)}
                g = {"w": torch.full((3000,), 0.01 * (k + 1), device="cuda", dtype=torch.bfloat16)}
                s = tx.init(p)
                for _ in range(20):
                    p, s = tx.step(p, s, g)
                torch.cuda.current_stream().synchronize()
                results[k] = (p, s)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors
    for k in range(4):
        p = {"w": torch.full((3000,), 1.0 + k, device="cuda", dtype=torch.bfloat16)}
        g = {"w": torch.full((3000,), 0.01 * (k + 1), device="cuda", dtype=torch.bfloat16)}
        s = ref.init(p)
        for _ in range(20):
            p, s = ref.step(p, s, g)
        _same((results[k][0], results[k][1].mu, results[k][1].nu), (p, s.mu, s.nu))


def test_trees_of_weights_through_the_codecs():
    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import tree

    p = _params(3)
    w = tree.tree_map(lambda x: torch.randn(x.shape, device="cuda"), p)
    for bits in (None, 24, 32):
        lp, ecc = fo.set_fp32_params(w, p, master_weight_bits=bits)
        want = tree.tree_map(lambda a, b: fo.split_leaf(a, narrow_dtype=b.dtype, master_weight_bits=bits), w, p)
        for a, b, (c, d) in zip(_leaves(lp), _leaves(ecc), tree.tree_leaves(want, is_leaf=lambda x: type(x) is tuple and isinstance(x[0], torch.Tensor))):
            _same((a, b), (c, d))
        back = fo.reconstruct_weights(lp, ecc)
        _same(back, tree.tree_map(fo.reconstruct_leaf, lp, ecc))
    with pytest.raises(ValueError):
        fo.reconstruct_weights(lp, {"a": ecc["a"]})


@pytest.mark.parametrize("group", [1, 8, 16, 32, 100, 256, 512])
def test_codecs_at_edges(group):
    import numpy as np
    import torch

    import flashoptim_jax_b200 as fo
    from oracle import flashoptim_oracle as O

    rng = np.random.default_rng(group)
    for n in (1, 7, 8, 2047, 2048, 2049, 3 * 2048 + 5):
        x = rng.normal(0, 1e-3, n).astype(np.float32)
        x[: n // 5] = 0
        for variance in (False, True):
            v = x * x if variance else x
            t = torch.from_numpy(np.concatenate([np.zeros(1, np.float32), v])).cuda()[1:]  # not 32-byte aligned
            for a in (t, t.clone()):
                q = (fo.quantize_variance if variance else fo.quantize_momentum)(a, group)
                want_q = (O.quantize_variance if variance else O.quantize_momentum)(v, group)
                assert np.array_equal(q.values.cpu().numpy(), want_q.values) and np.array_equal(q.scales.cpu().numpy(), want_q.scales)
                d = (fo.dequantize_variance if variance else fo.dequantize_momentum)(q, group)
                want = (O.dequantize_variance if variance else O.dequantize_momentum)(want_q, group)
                assert np.array_equal(d.cpu().numpy(), want)


@pytest.mark.parametrize("donate", [False, True])
@pytest.mark.parametrize("where", ["schedule", "selector"])
def test_callbacks_that_touch_the_trees(where, donate):
    """A schedule or a selector puts other storage under a parameter, or another tensor into the tree, while the step is being prepared: what
    is in the tree when the step is launched is stepped."""
    import torch

    import flashoptim_jax_b200 as fo

    trees = {}

    def touch(leaf_of):
        p = trees["params"]
        p["w"].data = p["w"].data.clone()
        if leaf_of == "b":
            p["b"] = p["b"].clone()
        del p

    kw = {}
    if where == "schedule":
        kw["learning_rate"] = lambda count: (touch("b"), 1e-2)[1]
    else:
        kw.update(learning_rate=1e-2, param_groups=[{"params": lambda path, leaf: (touch(path[0]), False)[1], "weight_decay": 0.5}])
    tx, ref = fo.flash_adamw(donate=donate, **kw), fo.flash_adamw(learning_rate=1e-2)
    make = lambda: {"b": torch.ones(33, device="cuda"), "w": torch.full((3000,), 0.5, device="cuda", dtype=torch.bfloat16)}
    p, q = make(), make()
    trees["params"] = p
    s, t = tx.init(p), ref.init(q)
    for k in range(5):
        g = _grads(q, k)
        trees["params"] = p
        p, s = tx.step(p, s, g)
        q, t = ref.step(q, t, g)
        if donate:
            p = dict(p)  # a container of its own for the next callback
        _same((p, s.mu, s.nu, s.ecc), (q, t.mu, t.nu, t.ecc))


def test_the_gil_is_released_around_launches():
    """Every call of the host extension into the library, with the library's function replaced by PyGILState_Check: 1, which reads as an
    invalid argument, where the calling thread holds the GIL."""
    import ctypes

    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import _lib, clipping

    host, lib = _lib.host(), _lib.lib()
    names = ("fo_step_ex", "fo_sq_norm_mixed", "fo_split_many", "fo_reconstruct_many", "fo_quantize_momentum", "fo_quantize_variance",
             "fo_dequantize_momentum", "fo_dequantize_variance", "fo_status_string", "fo_last_error")
    table = {name: ctypes.cast(getattr(lib, name), ctypes.c_void_p).value for name in names}
    check = ctypes.cast(ctypes.pythonapi.PyGILState_Check, ctypes.c_void_p).value
    p = {"w": torch.ones(64, device="cuda", dtype=torch.bfloat16)}
    steps = []
    for donate in (False, True):
        tx = fo.flash_adamw(donate=donate)
        q, s = p, tx.init(p)
        for _ in range(2):
            q, s = tx.step(q, s, p)
        steps.append((tx, q, s))
    x = torch.ones(64, device="cuda")
    codes = fo.quantize_momentum(x)
    lp, ecc = fo.set_fp32_params({"w": x}, p)
    host.bind({**table, **{name: check for name in names[:8]}}, fo.QuantizedArray)
    try:
        for tx, q, s in steps:
            tx.step(q, s, p)
        clipping.global_sq_norm(p)
        fo.set_fp32_params({"w": x}, p)
        fo.reconstruct_weights(lp, ecc)
        fo.quantize_momentum(x), fo.quantize_variance(x), fo.dequantize_momentum(codes), fo.dequantize_variance(codes)
    finally:
        host.bind(table, fo.QuantizedArray)


@contextlib.contextmanager
def _only_planned_steps(monkeypatch):
    from flashoptim_jax_b200 import _engine as eng

    def refuse(*a, **k):
        raise AssertionError("the general path took a step")

    with monkeypatch.context() as m:
        m.setattr(eng, "launch", refuse)
        yield


@pytest.mark.parametrize("donate", [False, True])
def test_learning_rates_written_before_every_step(donate, monkeypatch):
    import torch

    import flashoptim_jax_b200 as fo

    groups, plain = [[{"params": "bias", "learning_rate": 1e-2, "weight_decay": 0.0}, {"params": "a/w", "learning_rate": lambda c: 1e-3}] for _ in range(2)]
    tx, ref = fo.flash_lion(learning_rate=1e-4, param_groups=groups, donate=donate), fo.flash_lion(learning_rate=1e-4, param_groups=plain)
    p, q = _params(), _params()
    s, t = tx.init(p), ref.init(q)
    p, s = tx.step(p, s, _grads(q, 9))
    q, t = ref.step(q, t, _grads(q, 9))
    rates = [3e-2, 1, torch.tensor(2e-2), lambda c: 1e-2 * int(c), 0.0, 5e-3]
    grads = [_grads(_params(), k) for k in range(len(rates))]
    with _only_planned_steps(monkeypatch):
        for k, rate in enumerate(rates):
            groups[0]["learning_rate"], groups[1]["learning_rate"] = rate, rates[-1 - k]
            p, s = tx.step(p, s, grads[k])
    for k, rate in enumerate(rates):
        plain[0]["learning_rate"], plain[1]["learning_rate"] = rate, rates[-1 - k]
        with _general_path():
            q, t = ref.step(q, t, grads[k])
    _same((p, s.mu, s.ecc), (q, t.mu, t.ecc))


def test_markers_have_storage_of_their_own():
    """The 0-d zeros of leaves without an error-correction code: none shares memory, or a saved file, with another."""
    import torch

    import flashoptim_jax_b200 as fo

    w = {k: torch.ones(5, device="cuda") for k in "abc"}
    like = {"a": w["a"], "b": w["b"], "c": torch.empty(5, device="cuda", dtype=torch.bfloat16)}
    for bits, count in ((24, 2), (None, 3)):
        ecc = fo.set_fp32_params(w, like, master_weight_bits=bits)[1]
        markers = [e for e in ecc.values() if e.dim() == 0]
        assert len(markers) == count and all(e.dtype == torch.int32 and int(e) == 0 and e.untyped_storage().nbytes() == 4 for e in markers)
        assert len({e.data_ptr() for e in markers}) == count


def test_selectors_that_read_values():
    """Asked before the step and not after it; a donated step that changes the answer does not change what it used."""
    import torch

    import flashoptim_jax_b200 as fo

    asked = []

    def large(path, leaf):
        asked.append(path)
        return bool((leaf > 0.995).all())

    make = lambda: {"w": torch.ones(64, device="cuda", dtype=torch.bfloat16), "x": torch.ones(64, device="cuda")}
    results = []
    for donate in (False, True):
        tx = fo.flash_sgd(learning_rate=1e-2, momentum=0.0, donate=donate, param_groups=[{"params": large, "learning_rate": 2e-2}])
        p = make()
        s = tx.init(p)
        for _ in range(4):
            asked.clear()
            p, s = tx.step(p, s, {k: torch.ones_like(v) for k, v in p.items()})
            assert asked[-2:] == [("w",), ("x",)]  # (before them perhaps for a plan that did not fit)
        results.append(p)
    _same(*results)


@pytest.mark.parametrize("name", ["flash_adamw", "flash_lion", "flash_sgd"])
def test_a_step_that_cannot_be_planned_has_no_effect(name, monkeypatch):
    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import _lib

    def missing():
        raise _lib.NativeLibraryError("no extension")

    tx = getattr(fo, name)(donate=True)
    p = {"w": torch.ones(64, device="cuda", dtype=torch.bfloat16)}
    s = tx.init(p)
    before = [x.clone() for x in _leaves((p, s.mu))]
    with monkeypatch.context() as m:
        m.setattr(_lib, "host", missing)
        with pytest.raises(_lib.NativeLibraryError):
            tx.step(p, s, p)
    _same((p, s.mu), before)
    p, s = tx.step(p, s, {"w": torch.ones_like(p["w"])})
    assert int(s.count) == 1


def test_equal_keys_of_another_type_are_another_tree():
    import torch

    import flashoptim_jax_b200 as fo

    tx = fo.flash_lion(learning_rate=1e-2, param_groups=[{"params": "1", "learning_rate": 0.0}])
    w = torch.ones(64, device="cuda", dtype=torch.bfloat16)
    g, p = torch.ones_like(w), {1: w}
    s = tx.init(p)
    for _ in range(2):
        p, s = tx.step(p, s, {1: g})
    assert torch.equal(p[1], w)
    t = type(s)(s.count, *({True: x[1]} for x in (s.mu, s.ecc)))
    q, t = tx.step({True: p[1]}, t, {True: g})  # its path reads "True"
    assert type(next(iter(q))) is bool and not torch.equal(q[True], w)


class Checked(Pair):
    """A NamedTuple with a constructor of its own."""

    made = 0

    def __new__(cls, kernel, bias):
        Checked.made += 1
        return super().__new__(cls, kernel, bias)


class Plain(Pair):
    pass


def test_named_tuples_are_made_by_their_constructors():
    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import clipping

    for kind in (Checked, Plain):
        make = lambda: kind(torch.ones(64, device="cuda", dtype=torch.bfloat16), torch.ones(5, device="cuda"))
        tx, ref = fo.flash_lion(learning_rate=1e-2), fo.flash_lion(learning_rate=1e-2)
        p, q = make(), make()
        s, t = tx.init(p), ref.init(q)
        for k in range(3):
            g = kind(*(0.1 * (k + 1) * torch.ones_like(x) for x in q))
            Checked.made = 0
            p, s = tx.step(p, s, g)
            assert type(p) is kind and type(s.mu) is kind and (kind is Plain or Checked.made == 3)
            with _general_path():
                q, t = ref.step(q, t, g)
            _same((p, s.mu, s.ecc), (q, t.mu, t.ecc))
        sq = float(clipping.global_sq_norm(g))
        assert abs(sq - sum(float((x.double() ** 2).sum()) for x in g)) <= 1e-6 * sq
        w, ecc = fo.set_fp32_params(kind(*(x.float() for x in p)), p)
        assert type(w) is kind and type(ecc) is kind and type(fo.reconstruct_weights(w, ecc)) is kind


@pytest.mark.parametrize("donate", [False, True])
def test_ordered_and_default_dicts_are_planned(donate, monkeypatch):
    """Their order does not matter, and plain dicts come back, as from the general path."""
    import torch

    import flashoptim_jax_b200 as fo

    ordered = lambda x: collections.OrderedDict((k, collections.defaultdict(list, v) if isinstance(v, dict) else v) for k, v in reversed(x.items()))
    make = lambda: {"a": {"w": torch.ones(64, device="cuda", dtype=torch.bfloat16), "v": torch.ones(7, device="cuda")}, "b": torch.ones(5, device="cuda")}
    tx, ref = fo.flash_adamw(donate=donate), fo.flash_adamw()
    p, q = make(), make()
    s, t = tx.init(p), ref.init(q)
    grads = [_grads(make(), k) for k in range(4)]
    p, s = tx.step(p, s, grads[0])
    with _only_planned_steps(monkeypatch):
        for g in grads[1:]:
            p, s = tx.step(ordered(p), s, ordered(g))
            assert type(p) is dict and type(p["a"]) is dict and list(p) == ["a", "b"]
    with _general_path():
        for g in grads:
            q, t = ref.step(q, t, g)
    _same((p, s.mu, s.nu, s.ecc), (q, t.mu, t.nu, t.ecc))


@pytest.mark.parametrize("donate", [False, True])
def test_plans_of_several_tables_and_hyper_sets(donate, monkeypatch):
    """More leaves than a launch holds, and more hyper-parameter sets than a call takes, through a compiled plan."""
    import torch

    import flashoptim_jax_b200 as fo

    names = [f"{i:03d}" for i in range(700)]
    groups = [{"params": names[i::40], "learning_rate": 1e-3 * (i + 1), "weight_decay": 0.01 * i} for i in range(20)]
    rng = torch.Generator(device="cuda").manual_seed(0)
    make = lambda: {k: torch.full((1 + 37 * i % 2500,), 0.02 * (1 + i % 7), device="cuda", dtype=torch.bfloat16 if i % 5 else torch.float32) for i, k in enumerate(names)}
    tx, ref = fo.flash_adamw(param_groups=groups, donate=donate), fo.flash_adamw(param_groups=groups)
    p, q = make(), make()
    s, t = tx.init(p), ref.init(q)
    for k in range(3):
        g = {n: (torch.randn(x.shape, device="cuda", generator=rng) * 1e-2).to(x.dtype) for n, x in q.items()}
        with _only_planned_steps(monkeypatch) if k else contextlib.nullcontext():
            p, s = tx.step(p, s, g)
        with _general_path():
            q, t = ref.step(q, t, g)
        _same((p, s.mu, s.nu, s.ecc), (q, t.mu, t.nu, t.ecc))
