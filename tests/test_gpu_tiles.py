"""tile_kernel, bit for bit against the CPU oracle, where its tiles of 512 elements, its leaf tables and its copies can go wrong:
leaves that end around a tile or shorter than one, runs that begin inside a leaf, arrays that start off 32 bytes (parameters and
ECC then leave in two stores) or in the middle of a four-byte word (scales), every gradient dtype, weight decay added to the gradient."""

import numpy as np
import pytest

from oracle import c_oracle as C
from oracle import flashoptim_oracle as O
from tests import helpers as H
from tests.test_gpu_step_routes import G_NP, _step

pytestmark = pytest.mark.gpu

MANY = 148 * 8192 + 1  # more elements than go through piece_kernel alone (148 * 4096 here)
SIZES = (512, 511, 513, 255, 256, 257, 767, 768, 769, 1, 1023, 1025, 1536, 2047, 2048, 3072 + 511, 16 * 1024, 16 * 1024 + 512, 33 * 1024, 5)


def _moved(t, elems):
    """The same values `elems` elements further into an allocation."""
    import torch

    return None if t is None else torch.cat([t[:1].expand(elems), t])[elems:]


def _check(opt, pdt, ecc_bits, group, conv, gdt, sizes, *, max_norm=None, elsewhere=False, moved=None, **hyper):
    import torch

    from flashoptim_jax_b200 import _engine as eng

    rng = np.random.default_rng(sum(sizes) + group + gdt)
    refs = [H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, group) for n in sizes]
    refs[0].param[::97] = 0  # values outside the shortcuts' ranges
    place = (lambda leaf: H.LeafArrays(*[_moved(getattr(leaf, f), moved[f]) for f in leaf.fields()])) if moved else lambda leaf: leaf
    devs = [place(r.copy().to_device()) for r in refs]
    for t in (1, 2):
        grads = [H.make_grad(rng, n, 1e-2, G_NP[gdt], outliers=1e-3) for n in sizes]
        hp = H.hyper_tuple(opt, conv, t, lr=1e-3, wd=1e-2, **hyper)
        dev_g = [H.to_torch(g) for g in grads]
        sq = None
        if max_norm is not None:
            sq = eng.sq_norm_of(dev_g)
            grads = O.clip_by_global_norm(grads, max_norm, sq_norm=float(sq.cpu()))
        for g, r in zip(grads, refs):
            H.oracle_step(opt, g, r, C.STATE_QUANT, group, hp)
        outs = [place(H.LeafArrays(*[None if getattr(d, f) is None else torch.empty_like(getattr(d, f)) for f in d.fields()])) for d in devs] if elsewhere else None
        _step(opt, dev_g, devs, outs, C.STATE_QUANT, group, hp, pdt, gdt, ecc_bits, sq, max_norm or 0.0)
        torch.cuda.synchronize()
        devs = outs if elsewhere else devs
        for i, (d, r) in enumerate(zip(devs, refs)):
            H.assert_leaf_equal(d.to_host(), r, f"step {t} leaf {i} n={sizes[i]}")


def _kernels_of(call):
    """Names of the kernels that `call` launches."""
    import torch

    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
    kernels = {e.key for e in prof.key_averages()}
    if not any("kernel" in k for k in kernels):
        pytest.skip("the profiler records no kernels here")
    return kernels


@pytest.mark.parametrize("gdt", [0, 1, 2])
@pytest.mark.parametrize("opt,pdt,ecc_bits,group,conv,more", [
    (C.ADAM, 1, 16, 32, O.FUSED, {}), (C.ADAM, 2, 8, 256, O.FUSED, {}), (C.ADAM, 1, 8, 32, O.UNFUSED, {}), (C.ADAM, 0, 0, 16, O.FUSED, {}),
    (C.ADAM, 1, 0, 32, O.FUSED, dict(max_norm=0.5)), (C.ADAM, 2, 16, 32, O.FUSED, dict(elsewhere=True)), (C.ADAM, 1, 8, 8, O.FUSED, {}),
    (C.ADAM, 1, 16, 32, O.FUSED, dict(decoupled=False)), (C.LION, 1, 8, 32, O.FUSED, {}), (C.LION, 2, 16, 64, O.UNFUSED, {}),
    (C.LION, 0, 0, 32, O.FUSED, dict(max_norm=0.5)), (C.SGD, 1, 16, 32, O.FUSED, dict(nesterov=True)), (C.SGD, 2, 8, 128, O.FUSED, {}),
    (C.SGD, 0, 0, 32, O.FUSED, dict(decoupled=False)), (C.SGD, 1, 8, 32, O.FUSED, dict(elsewhere=True))])
def test_leaves_that_end_around_a_tile(opt, pdt, ecc_bits, group, conv, more, gdt):
    _check(opt, pdt, ecc_bits, group, conv, gdt, (MANY + 700,) + SIZES, **more)


@pytest.mark.parametrize("more", [{}, dict(max_norm=0.5), dict(elsewhere=True), dict(group=128), dict(conv=O.UNFUSED)])
@pytest.mark.parametrize("opt,pdt,ecc_bits,gdt", [(C.ADAM, 1, 16, 1), (C.ADAM, 2, 8, 0), (C.ADAM, 0, 0, 0), (C.SGD, 1, 8, 1), (C.SGD, 2, 0, 1)])
def test_decay_added_to_the_gradient(opt, pdt, ecc_bits, gdt, more):
    """A weight decay that is added to the gradient beside every feature, by tile_kernel as without it."""
    more = dict(dict(group=32, conv=O.FUSED), **more)
    group, conv = more.pop("group"), more.pop("conv")
    kernels = _kernels_of(lambda: _check(opt, pdt, ecc_bits, group, conv, gdt, (MANY + 700,) + SIZES, decoupled=False, **more))
    assert any("tile_kernel" in k for k in kernels) and not any("step_kernel" in k for k in kernels), kernels


@pytest.mark.parametrize("opt,pdt,ecc_bits", [(C.ADAM, 1, 16), (C.LION, 2, 8), (C.SGD, 0, 0)])
def test_groups_of_8_have_a_kernel_of_their_own(opt, pdt, ecc_bits):
    kernels = _kernels_of(lambda: _check(opt, pdt, ecc_bits, 8, O.FUSED, 1, (MANY + 6143 * 3, 8 * 6144, 7)))
    main = {k for k in kernels if "step_kernel" in k or "tile_kernel" in k}
    assert len(main) == 1 and f"step_kernel<{opt}, {pdt}, {ecc_bits}, 0, 4>" in main.pop(), kernels


@pytest.mark.parametrize("offset,scale_offset", [(8, 1), (16, 2), (8, 2), (24, 3)])
@pytest.mark.parametrize("opt,pdt,ecc_bits,elsewhere", [(C.ADAM, 1, 16, False), (C.ADAM, 2, 8, True), (C.LION, 1, 16, True), (C.SGD, 0, 0, False)])
def test_arrays_off_the_alignment_of_the_wide_accesses(opt, pdt, ecc_bits, elsewhere, offset, scale_offset):
    moved = {"param": offset // (2 if pdt == 0 else 1), "ecc": offset * 2 if ecc_bits == 8 else offset, "mu": 16, "nu": 48, "mu_scales": scale_offset,
             "nu_scales": 2}
    _check(opt, pdt, ecc_bits, 32, O.FUSED, 0, (MANY + 700, 4096, 1536), elsewhere=elsewhere, moved=moved)


def test_tables_of_many_leaves_and_several_runs_per_block():
    rng = np.random.default_rng(5)
    _check(C.ADAM, 1, 8, 32, O.FUSED, 1, tuple(int(x) for x in rng.integers(500, 30000, 330)))
    _check(C.LION, 1, 8, 32, O.FUSED, 1, (148 * 512 * 300 + 1024, 700 * 1024 + 512, 3 * 1024))  # more than 256 tiles per block


@pytest.mark.parametrize("opt,pdt,ecc_bits,group,more", [
    (C.ADAM, 1, 16, 32, {}), (C.ADAM, 0, 0, 32, dict(decoupled=False, wd=0.0)), (C.LION, 1, 16, 32, {}), (C.LION, 2, 8, 128, {}), (C.LION, 0, 0, 32, {}),
    (C.SGD, 1, 8, 32, {}), (C.SGD, 2, 16, 256, dict(nesterov=True)), (C.SGD, 0, 0, 32, {}), (C.SGD, 0, 0, 32, dict(decoupled=False, wd=0.0)),
    (C.SGD, 1, 8, 32, dict(lr=-1e-3, momentum=-0.9)), (C.LION, 2, 8, 32, dict(lr=-1e-3))])
def test_rows_at_rest_in_parts_of_tiles(opt, pdt, ecc_bits, group, more):
    """Rows without gradients that begin and end inside tiles and halves of tiles, with zeros of both signs and infinities among
    their parameters."""
    import torch

    rng = np.random.default_rng(opt * 10 + pdt)
    n = MANY + 5000
    p = rng.normal(0, 0.02, n).astype(np.float32)
    p[::301], p[7::401] = 0.0, -0.0
    if pdt != 1:
        p[5::70001] = np.inf
    ref = H.fresh_leaf(p.astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, group)
    dev = ref.copy().to_device()
    kw = dict(dict(lr=1e-3, wd=1e-2), **more)
    for t in (1, 2):
        g = H.make_grad(rng, n, 1e-2, H.BF16)
        for start, length in ((0, 512), (5 * 512 + 256, 256), (9000, 700), (20000, 1408), (30001, 4099), (n - 3000, 3000)):
            g[start:start + length] = 0
            g[start:start + length:3] = -0.0
        hp = H.hyper_tuple(opt, O.FUSED, t, **kw)
        H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
        _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, group, hp, pdt, 1, ecc_bits)
        torch.cuda.synchronize()
        got = dev.to_host()
        both = np.isnan(got.param.astype(np.float32)) & np.isnan(ref.param.astype(np.float32))
        got.param[both] = ref.param[both]  # (whichever NaN it is)
        H.assert_leaf_equal(got, ref, f"step {t}")


def _but_for_nans(got, ref, group, at):
    """`got` with what NaNs leave open made that of `ref`: which NaN a parameter is, and, where the elements `at` have NaN moments, the scales of
    their groups (any size but 32: NaN, which is checked here; of 32 elements that of the others) and the codes beside them."""
    both = np.isnan(got.param.astype(np.float32)) & np.isnan(ref.param.astype(np.float32))
    got.param[both] = ref.param[both]
    if group != 32:
        hit = np.unique(at // group)
        for scales, codes in (("mu_scales", "mu"), ("nu_scales", "nu")):
            if getattr(ref, scales) is not None:
                assert np.isnan(getattr(got, scales)[hit]).all()
                getattr(got, scales)[hit] = getattr(ref, scales)[hit]
                inside = np.isin(np.arange(ref.param.size) // group, hit)
                getattr(got, codes)[inside] = getattr(ref, codes)[inside]
    return got


@pytest.mark.parametrize("n", [1000, MANY + 700])
@pytest.mark.parametrize("decay", [dict(decoupled=False, wd=0.0), dict(decoupled=False, wd=1e-2), dict(wd=1e-2)])
@pytest.mark.parametrize("opt,pdt,group", [(C.ADAM, 1, 32), (C.ADAM, 2, 64), (C.ADAM, 0, 32), (C.SGD, 1, 16), (C.SGD, 2, 32), (C.SGD, 0, 128), (C.LION, 2, 32)])
def test_parameters_without_codes_that_are_not_finite(opt, pdt, group, decay, n):
    """Infinities and NaNs among parameters without error-correction codes: a decay that is added to the gradient makes the element's
    moments NaN, a decay of zero too."""
    rng = np.random.default_rng(n + opt)
    p = rng.normal(0, 0.02, n).astype(np.float32)
    for value in (np.inf, -np.inf, np.nan):
        p[rng.integers(0, n, 1 + n // 3000)] = value
    ref = H.fresh_leaf(p.astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, 0, group)
    dev = ref.copy().to_device()
    g = H.make_grad(rng, n, 1e-2, H.BF16)
    hp = H.hyper_tuple(opt, O.FUSED, 1, **dict(dict(lr=1e-3), **decay))
    H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
    _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, group, hp, pdt, 1, 0)
    odd = np.isnan(p) if decay["wd"] != 0.0 else ~np.isfinite(p)  # (a decay of infinity that is not zero is an infinity)
    at = np.flatnonzero(odd) if opt != C.LION and "decoupled" in decay else np.empty(0, dtype=np.int64)
    H.assert_leaf_equal(_but_for_nans(dev.to_host(), ref, group, at), ref, f"n={n}")


@pytest.mark.parametrize("n", [1024, 3000, MANY + 700])
@pytest.mark.parametrize("opt,pdt,ecc_bits", [(C.ADAM, 1, 0), (C.ADAM, 2, 0), (C.ADAM, 0, 0), (C.SGD, 1, 0), (C.SGD, 2, 0), (C.SGD, 0, 0), (C.ADAM, 1, 8), (C.SGD, 2, 16)])
def test_parameters_at_rest_that_are_not_finite(opt, pdt, ecc_bits, n):
    """The same in rows without gradients, under a decay of zero that is added to the gradient: no rows at rest, in pieces and in tiles."""
    rng = np.random.default_rng(n + opt)
    p = rng.normal(0, 0.02, n).astype(np.float32)
    at = np.unique(rng.integers(0, n, 3 + n // 3000))
    p[at] = rng.choice([np.inf, -np.inf], at.size) if ecc_bits else rng.choice([np.inf, -np.inf, np.nan], at.size)
    ref = H.fresh_leaf(p.astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, 32)
    dev = ref.copy().to_device()
    g = np.zeros(n, dtype=H.BF16)
    g[::3] = -0.0
    hp = H.hyper_tuple(opt, O.FUSED, 1, lr=1e-3, decoupled=False, wd=0.0)
    for t in (1, 2):
        H.oracle_step(opt, g, ref, C.STATE_QUANT, 32, hp)
        _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, 32, hp, pdt, 1, ecc_bits)
        H.assert_leaf_equal(_but_for_nans(dev.to_host(), ref, 32, at), ref, f"n={n} step {t}")


@pytest.mark.parametrize("n", [1024, MANY + 700])
@pytest.mark.parametrize("lr", [-0.0, -1e-3, np.inf])
@pytest.mark.parametrize("opt", [C.ADAM, C.LION, C.SGD])
def test_rows_at_rest_under_learning_rates_that_change_them(opt, lr, n):
    """A parameter of -0 becomes +0 under a learning rate with a sign, every parameter a NaN under an infinite one."""
    ref = H.fresh_leaf(np.where(np.arange(n) % 3 == 0, -0.0, 0.5).astype(np.float32), opt, C.STATE_QUANT, 0, 32)
    dev = ref.copy().to_device()
    g = np.zeros(n, dtype=np.float32)
    hp = H.hyper_tuple(opt, O.FUSED, 1, lr=lr, wd=1e-2)
    H.oracle_step(opt, g, ref, C.STATE_QUANT, 32, hp)
    _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, 32, hp, 0, 0, 0)
    H.assert_leaf_equal(_but_for_nans(dev.to_host(), ref, 32, np.empty(0, dtype=np.int64)), ref, f"n={n} lr={lr}")


@pytest.mark.parametrize("n", [3000, MANY + 700])
@pytest.mark.parametrize("opt,pdt,ecc_bits,group,conv", [
    (C.ADAM, 1, 16, 32, O.FUSED), (C.ADAM, 1, 8, 128, O.FUSED), (C.ADAM, 2, 8, 32, O.UNFUSED), (C.ADAM, 0, 0, 16, O.FUSED), (C.LION, 1, 8, 32, O.FUSED),
    (C.LION, 2, 16, 256, O.UNFUSED), (C.SGD, 1, 16, 32, O.FUSED), (C.SGD, 2, 8, 64, O.FUSED)])
def test_scattered_odd_values(opt, pdt, ecc_bits, group, conv, n):
    """Single elements outside the shortcuts' ranges among ordinary ones, which the repairs leave alone: parameters of zero, next to it and near
    the largest, elements that never see a gradient, gradients whose square overflows."""
    rng = np.random.default_rng(n + opt + group)
    pick = lambda: rng.integers(0, n, 1 + n // 300)  # noqa: E731
    p = rng.normal(0, 0.02, n).astype(np.float32)
    for value in (0.0, -0.0, 1e-38, -3e-31, 6e4, -6e4):
        p[pick()] = value
    if pdt != 2:
        p[pick()] = 2e38
    never, huge = pick(), pick()
    ref = H.fresh_leaf(p.astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, group)
    dev = ref.copy().to_device()
    for t in (1, 2):
        g = H.make_grad(rng, n, 1e-2, np.float32)
        if t == 2:  # (the fp16 scales of their groups are infinite then)
            g[huge] = 1e20
        g[never] = 0
        hp = H.hyper_tuple(opt, conv, t, lr=1e-3, wd=1e-2)
        H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
        _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, group, hp, pdt, 0, ecc_bits)
        H.assert_leaf_equal(dev.to_host(), ref, f"step {t}")


@pytest.mark.parametrize("first", ["outside", "inside"])
@pytest.mark.parametrize("pdt,ecc_bits,group,max_norm,elsewhere", [(1, 16, 32, None, False), (2, 8, 32, 0.5, False), (0, 0, 128, None, False), (1, 8, 32, None, True)])
def test_device_scalars_outside_the_proven_range_beside_ordinary_leaves(pdt, ecc_bits, group, max_norm, elsewhere, first):
    """Leaves whose eps lies outside the range of the reciprocal shortcut, which tile_kernel learns while it runs (the scalars are the device's), in
    turn with ordinary ones: first tiles that were asked for ahead and are dropped, later leaves in the same slots, ragged ends of both."""
    import torch

    from flashoptim_jax_b200 import _engine as eng

    rng = np.random.default_rng(group + pdt)
    sizes = (148 * 4096 + 700, 40 * 1024 + 9, 300 * 1024 + 513, 511, 64 * 1024, 700, 90 * 1024 + 255)
    refs = [H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), C.ADAM, C.STATE_QUANT, ecc_bits, group) for n in sizes]
    devs = [r.copy().to_device() for r in refs]
    hyper_of = [(i + (first == "inside")) % 2 for i in range(len(sizes))]  # 0: outside
    for t in (1, 2):
        hps = [H.hyper_tuple(C.ADAM, O.FUSED, t, lr=1e-3, wd=1e-2, eps=eps) for eps in (1e-13, 1e-8)]
        scalars = torch.tensor([hps[0][0], hps[0][7], hps[0][8]], device="cuda")
        grads = [H.make_grad(rng, n, 1e-2, H.BF16) for n in sizes]
        dev_g, sq = [H.to_torch(g) for g in grads], None
        if max_norm is not None:
            sq = eng.sq_norm_of(dev_g)
            grads = O.clip_by_global_norm(grads, max_norm, sq_norm=float(sq.cpu()))
        for g, r, h in zip(grads, refs, hyper_of):
            H.oracle_step(C.ADAM, g, r, C.STATE_QUANT, group, hps[h])
        outs = [H.LeafArrays(*[None if getattr(d, f) is None else torch.empty_like(getattr(d, f)) for f in d.fields()]) for d in devs] if elsewhere else None
        H.abi_step(C.ADAM, dev_g, devs, C.STATE_QUANT, group, [hp + (scalars.data_ptr(),) for hp in hps], hyper_of, pdt, 1, ecc_bits,
                   grad_sq_norm=sq, max_grad_norm=max_norm or 0.0, outs=outs)
        torch.cuda.synchronize()
        devs = outs if elsewhere else devs
        for i, (d, r) in enumerate(zip(devs, refs)):
            H.assert_leaf_equal(d.to_host(), r, f"step {t} leaf {i} n={sizes[i]}")


@pytest.mark.parametrize("opt,ecc_bits,group,gdt,more", [
    (C.ADAM, 16, 32, 1, {}), (C.ADAM, 8, 32, 0, {}), (C.ADAM, 8, 128, 1, dict(conv=O.UNFUSED)), (C.ADAM, 16, 32, 1, dict(max_norm=0.5)),
    (C.ADAM, 8, 32, 1, dict(max_norm=0.5, lr=20.0)), (C.ADAM, 8, 32, 1, dict(lr=0.0)), (C.ADAM, 16, 32, 1, dict(lr=1e-12, eps=1e-12)),
    (C.ADAM, 8, 32, 1, dict(wd=4e3)), (C.ADAM, 8, 32, 1, dict(b1=1e-9, max_norm=0.5)), (C.ADAM, 16, 32, 1, dict(b1=0.0, max_norm=0.5)), (C.ADAM, 8, 32, 1, dict(decoupled=False)),
    (C.ADAM, 8, 32, 0, dict(elsewhere=True)), (C.ADAM, 8, 32, 1, dict(lr=20.0, eps=1e-12)), (C.ADAM, 16, 32, 0, dict(lr=50.0, max_norm=0.5, eps=1e-12)),
    (C.ADAM, 8, 32, 1, dict(max_norm=-300.0)), (C.ADAM, 16, 32, 1, dict(max_norm=-3e5, lr=1e-8)), (C.ADAM, 8, 32, 0, dict(max_norm=-300.0)), (C.SGD, 8, 32, 1, dict(max_norm=-300.0)),
    (C.ADAM, 8, 32, 1, dict(lr=1e-15, eps=1.0)), (C.ADAM, 16, 32, 1, dict(lr=1e-18, eps=1e-6, max_norm=0.5)), (C.LION, 16, 32, 1, dict(lr=1e-20)), (C.SGD, 16, 32, 1, dict(lr=1e-18)), (C.LION, 8, 32, 1, {}), (C.LION, 16, 64, 0, dict(conv=O.UNFUSED)), (C.LION, 8, 32, 1, dict(wd=4e3)),
    (C.SGD, 8, 32, 1, {}), (C.SGD, 16, 32, 0, dict(nesterov=True)), (C.SGD, 8, 32, 1, dict(lr=1e-9))])
def test_parameters_and_gradients_at_the_edges_of_the_first_pass(opt, ecc_bits, group, gdt, more):
    """bf16 parameters of every power of two, and next to it, from the smallest to the largest, some of which the update crosses, beside tiny
    gradients: alone in their tile and many in one."""
    import torch

    from flashoptim_jax_b200 import _engine as eng

    kw = dict(dict(lr=1e-3, wd=1e-2), **more)
    conv, max_norm, elsewhere = kw.pop("conv", O.FUSED), kw.pop("max_norm", None), kw.pop("elsewhere", False)
    rng = np.random.default_rng(opt * 100 + ecc_bits + gdt + len(more))
    n = 148 * 8192 + 700
    p = rng.normal(0, 0.02, n).astype(np.float32)
    edge = rng.random(n) < np.where(np.arange(n) < n // 2, 1 / 1000, 1 / 3)
    exponent = rng.integers(-133, 120 if kw.get("decoupled", True) else 10, n)  # (a decay in the gradient: fp16 scales of the moments stay finite)
    near = rng.random(n) < 0.5  # next to where the checks lie
    exponent[near] = rng.choice([-126, -101, -100, -99, -76, -75, -70, -69, -68, -67, -66, -64, -57, -56, -55, -50, -49, -48, -47, -38, -37, -36, -35, -34, -31, 0, 1, 2], int(near.sum()))
    edges = np.ldexp(rng.choice([1.0, 1.0 - 2.0**-8, 1.0 + 2.0**-7], n), exponent) * rng.choice([-1.0, 1.0], n)
    p[edge] = edges[edge].astype(np.float32)
    ref = H.fresh_leaf(p.astype(H.BF16), opt, C.STATE_QUANT, ecc_bits, group)
    dev = ref.copy().to_device()
    for t in (1, 2, 3):
        g = H.make_grad(rng, n, 1e-2, np.float32)
        tiny = rng.random(n) < 1 / 500
        g[tiny] = np.ldexp(rng.choice([-1.0, 1.0], int(tiny.sum())), rng.integers(-140, -20, int(tiny.sum())))
        g = g.astype(G_NP[gdt])
        hp = H.hyper_tuple(opt, conv, t, **kw)
        dev_g, sq = [H.to_torch(g)], None
        if max_norm is not None:
            sq = eng.sq_norm_of(dev_g)
            g = O.clip_by_global_norm([g], max_norm, sq_norm=float(sq.cpu()))[0]
        H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
        outs = [H.LeafArrays(*[None if getattr(dev, f) is None else torch.empty_like(getattr(dev, f)) for f in dev.fields()])] if elsewhere else None
        _step(opt, dev_g, [dev], outs, C.STATE_QUANT, group, hp, 1, gdt, ecc_bits, sq, max_norm or 0.0)
        torch.cuda.synchronize()
        dev = outs[0] if elsewhere else dev
        got = dev.to_host()
        both = np.isnan(got.param.astype(np.float32)) & np.isnan(ref.param.astype(np.float32))
        got.param[both] = ref.param[both]  # (whichever NaN it is)
        H.assert_leaf_equal(got, ref, f"step {t}")


@pytest.mark.parametrize("n", [1000, MANY + 700])
@pytest.mark.parametrize("conv", [O.FUSED, O.UNFUSED])
@pytest.mark.parametrize("factors", [dict(b1=np.nan, omb1=np.nan), dict(b1=np.nan), dict(omb1=np.nan), dict(b1=np.inf), dict(omb1=-np.inf), dict(b1=3e38, omb1=-3e38)])
@pytest.mark.parametrize("pdt,ecc_bits,group", [(1, 8, 32), (1, 16, 8), (2, 16, 64), (0, 0, 32)])
def test_lion_under_factors_that_are_not_finite(pdt, ecc_bits, group, factors, conv, n):
    """Factors that make the direction a NaN, and leave the moment what it is: so becomes the parameter, in pieces and in the first pass of tiles."""
    rng = np.random.default_rng(n + group)
    ref = H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), C.LION, C.STATE_QUANT, ecc_bits, group)
    dev = ref.copy().to_device()
    hp = list(H.hyper_tuple(C.LION, conv, 1, lr=1e-3, wd=1e-2))
    for t in (1, 2):
        g = H.make_grad(rng, n, 5e4, np.float32)
        g[::50] = 0
        if t == 2:  # (the first step gives moments)
            hp[2], hp[4] = np.float32(factors.get("b1", hp[2])), np.float32(factors.get("omb1", hp[4]))
        H.oracle_step(C.LION, g, ref, C.STATE_QUANT, group, hp)
        _step(C.LION, [H.to_torch(g)], [dev], None, C.STATE_QUANT, group, hp, pdt, 0, ecc_bits)
        H.assert_leaf_equal(_but_for_nans(dev.to_host(), ref, 32, np.empty(0, dtype=np.int64)), ref, f"step {t}")
    assert conv is O.UNFUSED or np.isnan(ref.param.astype(np.float32)).any()


def _in_turn(opt, ecc_bits, g, start, **runs):
    """ms that 20 steps take from the parameters start[name] with (hyper-parameters, square of the norm, limit) of runs[name], the smallest of nine, in turn."""
    import torch

    n, best = g.numel(), {}
    empty = H.fresh_leaf(np.zeros(0, H.BF16), opt, C.STATE_QUANT, ecc_bits)
    state = lambda a: None if a is None else torch.zeros(n // 32 if a.dtype == np.float16 else n, device="cuda", dtype=H.to_torch(a).dtype)  # noqa: E731
    leaves = {name: H.LeafArrays(start[name].clone(), *[state(getattr(empty, f)) for f in empty.fields()[1:]]) for name in runs}
    for _ in range(9):
        for name, (hp, sq, limit) in runs.items():
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            begin.record()
            for _ in range(20):
                _step(opt, [g], [leaves[name]], None, C.STATE_QUANT, 32, hp, 1, 1, ecc_bits, sq, limit)
            end.record()
            end.synchronize()
            best[name] = min(best.get(name, 1e9), begin.elapsed_time(end))
    return best


def _normal(n, sigma, seed):
    import torch

    return (torch.randn(n, device="cuda", generator=torch.Generator("cuda").manual_seed(seed)) * sigma).bfloat16()


@pytest.mark.parametrize("opt,lr,eps", [(C.ADAM, 1e-14, 1e-8), (C.ADAM, 20.0, 1e-12), (C.LION, 1e-14, 0.0), (C.SGD, 1e-14, 0.0)])
@pytest.mark.parametrize("ecc_bits", [8, 16])
def test_small_parameters_and_large_rates_take_the_first_pass(opt, ecc_bits, lr, eps):
    """A leaf a tenth of which is 1e-10 (as a matrix that started at zero, or pruned weights), or whose learning rate is large, against the same leaf without:
    not slower by more than half (repaired it takes twice as long and more)."""
    n = 1 << 24
    p, kw = _normal(n, 0.02, opt), dict(eps=eps) if opt == C.ADAM else {}
    odd = p.clone()
    if lr < 1:
        odd[::10] = 1e-10
    best = _in_turn(opt, ecc_bits, _normal(n, 1e-3, 9), dict(plain=p, odd=odd), plain=(H.hyper_tuple(opt, O.FUSED, 1, lr=1e-14, wd=1e-2, **kw), None, 0.0),
                    odd=(H.hyper_tuple(opt, O.FUSED, 1, lr=lr, wd=1e-2 if lr < 1 else 0.0, **kw), None, 0.0))
    assert best["odd"] <= 1.5 * best["plain"], best


@pytest.mark.parametrize("opt", [C.ADAM, C.LION, C.SGD])
def test_limits_below_zero_take_the_first_pass(opt):
    """Clipping to a limit below zero (gradients are turned round), which is larger than the norm, against one above it."""
    from flashoptim_jax_b200 import _engine as eng

    p, g = _normal(1 << 24, 0.02, opt), _normal(1 << 24, 1e-3, 9)
    hp, sq = H.hyper_tuple(opt, O.FUSED, 1, lr=1e-3), eng.sq_norm_of([g])
    best = _in_turn(opt, 8, g, dict(above=p, below=p), above=(hp, sq, 1.0), below=(hp, sq, -100.0))
    assert best["below"] <= 1.5 * best["above"], best
