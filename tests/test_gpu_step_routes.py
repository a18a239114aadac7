"""The routes a call can take through the step kernels, bit for bit against the CPU oracle: whole tiles through tile_kernel (quantized moments,
problems above 148 * 4096 elements), whole chunks through step_kernel (the rest, above 148 * 8192) with what they leave in pieces of 1024, small problems in pieces alone; groups of
8 to 256, parameters handed back as old + lp(new - old), results written elsewhere, clipping, and combinations."""

import ctypes

import ml_dtypes
import numpy as np
import pytest

from oracle import c_oracle as C
from oracle import flashoptim_oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu

MAIN = 148 * 8192 + 5 * 6144  # above the limit for every chunk size (2048, 4096, 6144)
G_NP = {0: np.float32, 1: ml_dtypes.bfloat16, 2: np.float16}


def _step(opt, grads, leaves, outs, state, group, hp, pdt, gdt, ecc_bits, sq=None, max_norm=0.0):
    from flashoptim_jax_b200 import _lib

    L = (_lib.FoLeaf * len(leaves))()
    X = (_lib.FoLeafOut * len(leaves))()
    for i, (g, lf) in enumerate(zip(grads, leaves)):
        L[i].grad, L[i].n, L[i].hyper = g.data_ptr(), lf.param.numel(), 0
        for name in lf.fields():
            t = getattr(lf, name)
            setattr(L[i], name, None if t is None else t.data_ptr())
            if outs is not None and t is not None:
                setattr(X[i], name, getattr(outs[i], name).data_ptr())
    hy = _lib.FoHyper()
    for k, name in enumerate(("lr", "wd", "b1", "b2", "one_minus_b1", "one_minus_b2", "eps", "bc1", "bc2")):
        setattr(hy, name, float(hp[k]))
    hy.flags = int(hp[9])
    d = _lib.FoStepDesc(struct_size=ctypes.sizeof(_lib.FoStepDesc), opt=opt, param_dtype=pdt, grad_dtype=gdt, ecc_bits=ecc_bits,
                        state=state, group_size=group, n_leaves=len(leaves), n_hypers=1, leaves=ctypes.cast(L, ctypes.c_void_p),
                        hypers=ctypes.cast(ctypes.pointer(hy), ctypes.c_void_p))
    more = _lib.FoStepMore(struct_size=ctypes.sizeof(_lib.FoStepMore), outs=None if outs is None else ctypes.cast(X, ctypes.c_void_p))
    if sq is not None:
        d.grad_sq_norm, d.max_grad_norm = sq.data_ptr(), max_norm
    _lib.check(_lib.lib().fo_step_ex(ctypes.byref(d), ctypes.byref(more), 0))


def _run(opt, pdt, ecc_bits, state, group, conv, sizes, *, gdt=1, elsewhere=False, max_norm=None, offset=0, steps=3):
    import torch

    from flashoptim_jax_b200 import _engine as eng

    rng = np.random.default_rng(sum(sizes) + group)
    refs = [H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), opt, state, ecc_bits, group) for n in sizes]
    for r in refs:
        r.param[: r.param.size // 50] = 0  # values outside the shortcuts' ranges
    devs = [r.copy().to_device() for r in refs]
    if offset:  # a leaf that does not start on a 16-byte boundary
        for d in devs:
            d.param = torch.cat([d.param[:offset], d.param])[offset:]
    for t in range(1, steps + 1):
        grads = [H.make_grad(rng, n, 1e-2, G_NP[gdt], outliers=1e-3) for n in sizes]
        for g in grads:
            g[: g.size // 3: 7] = 0
        hp = H.hyper_tuple(opt, conv, t, lr=1e-3, wd=1e-2)
        dev_g = [H.to_torch(g) for g in grads]
        sq = None
        if max_norm is not None:
            sq = eng.sq_norm_of(dev_g)
            grads = O.clip_by_global_norm(grads, max_norm, sq_norm=float(sq.cpu()))
        for g, r in zip(grads, refs):
            H.oracle_step(opt, g, r, state, group, hp)
        old = [H.LeafArrays(*[None if getattr(d, f) is None else getattr(d, f).clone() for f in d.fields()]) for d in devs] if elsewhere else None
        outs = [H.LeafArrays(*[None if getattr(d, f) is None else torch.empty_like(getattr(d, f)) for f in d.fields()]) for d in devs] if elsewhere else None
        _step(opt, dev_g, devs, outs, state, group, hp, pdt, gdt, ecc_bits, sq, max_norm or 0.0)
        torch.cuda.synchronize()
        if elsewhere:
            for a, b in zip(devs, old):  # the inputs are left alone
                H.assert_leaf_equal(a.to_host(), b.to_host(), f"inputs of step {t}")
            devs = outs
        for i, (d, r) in enumerate(zip(devs, refs)):
            H.assert_leaf_equal(d.to_host(), r, f"step {t} leaf {i} n={sizes[i]}")


@pytest.mark.parametrize("n", [MAIN, MAIN + 1, MAIN + 1023 * 3 + 5])
@pytest.mark.parametrize("opt,pdt,ecc_bits,state", [(C.ADAM, 1, 16, C.STATE_QUANT), (C.ADAM, 2, 8, C.STATE_QUANT), (C.ADAM, 0, 0, C.STATE_QUANT),
                                                    (C.ADAM, 1, 8, C.STATE_FULL), (C.LION, 1, 8, C.STATE_QUANT), (C.LION, 2, 16, C.STATE_FULL),
                                                    (C.SGD, 1, 16, C.STATE_QUANT), (C.SGD, 0, 0, C.STATE_FULL), (C.SGD, 2, 8, C.STATE_NONE)])
def test_whole_chunks_and_their_rest(opt, pdt, ecc_bits, state, n):
    _run(opt, pdt, ecc_bits, state, 32, O.FUSED, [n, 77], steps=2)


@pytest.mark.parametrize("group", [8, 16, 64, 128, 256])
@pytest.mark.parametrize("opt,pdt,ecc_bits", [(C.ADAM, 1, 16), (C.LION, 2, 8), (C.SGD, 0, 0)])
def test_group_sizes(opt, pdt, ecc_bits, group):
    _run(opt, pdt, ecc_bits, C.STATE_QUANT, group, O.FUSED, [MAIN + group + 3], gdt=0, steps=2)
    _run(opt, pdt, ecc_bits, C.STATE_QUANT, group, O.FUSED, [1, 7, group, group + 1, 1023, 1024, 1025, 5 * 1024 - group - 1])


@pytest.mark.parametrize("pdt,ecc_bits,state", [(1, 8, C.STATE_QUANT), (1, 16, C.STATE_FULL), (2, 0, C.STATE_QUANT), (0, 0, C.STATE_QUANT)])
def test_parameter_handed_back_as_a_delta(pdt, ecc_bits, state):
    _run(C.ADAM, pdt, ecc_bits, state, 32, O.UNFUSED, [MAIN + 1029], steps=2)
    _run(C.ADAM, pdt, ecc_bits, state, 32, O.UNFUSED, [3, 1024, 2047])


@pytest.mark.parametrize("opt,pdt,ecc_bits,state,group,conv", [
    (C.ADAM, 1, 8, C.STATE_QUANT, 32, O.FUSED), (C.ADAM, 1, 16, C.STATE_QUANT, 64, O.UNFUSED), (C.ADAM, 0, 0, C.STATE_FULL, 32, O.FUSED),
    (C.LION, 2, 16, C.STATE_QUANT, 32, O.FUSED), (C.SGD, 1, 0, C.STATE_NONE, 32, O.FUSED), (C.SGD, 1, 8, C.STATE_QUANT, 40, O.FUSED)])
def test_results_elsewhere(opt, pdt, ecc_bits, state, group, conv):
    _run(opt, pdt, ecc_bits, state, group, conv, [MAIN + 517, 33], elsewhere=True, steps=2)
    _run(opt, pdt, ecc_bits, state, group, conv, [1, 1000, 4096], elsewhere=True)
    _run(opt, pdt, ecc_bits, state, group, conv, [1500], elsewhere=True, offset=1)  # scalar path


@pytest.mark.parametrize("gdt", [0, 1, 2])
@pytest.mark.parametrize("max_norm", [0.5, 1e6])
def test_clipping_on_whole_chunks(gdt, max_norm):
    _run(C.ADAM, 1, 16, C.STATE_QUANT, 32, O.FUSED, [MAIN + 100, 2048], gdt=gdt, max_norm=max_norm, steps=2)
    _run(C.LION, 1, 8, C.STATE_QUANT, 64, O.FUSED, [MAIN], gdt=gdt, max_norm=max_norm, elsewhere=True, steps=2)


def test_many_leaves_need_several_tables():
    rng = np.random.default_rng(3)
    sizes = [int(x) for x in rng.integers(1, 9000, 500)]
    _run(C.ADAM, 1, 8, C.STATE_QUANT, 32, O.FUSED, sizes, steps=2)
    _run(C.ADAM, 1, 8, C.STATE_QUANT, 64, O.FUSED, sizes, steps=1, elsewhere=True)


@pytest.mark.parametrize("n", [1000, MAIN + 700])
@pytest.mark.parametrize("pdt,ecc_bits,state,group,conv", [
    (1, 16, C.STATE_QUANT, 32, O.FUSED), (0, 0, C.STATE_QUANT, 128, O.FUSED), (2, 8, C.STATE_QUANT, 16, O.UNFUSED), (1, 8, C.STATE_QUANT, 64, O.FUSED),
    (1, 8, C.STATE_FULL, 32, O.UNFUSED), (0, 0, C.STATE_FULL, 32, O.FUSED), (2, 16, C.STATE_FULL, 32, O.FUSED)])
def test_squares_that_overflow(pdt, ecc_bits, state, group, conv, n):
    """Gradients of 1e20: the second moment is an infinity and the update zero, for those elements alone."""
    rng = np.random.default_rng(n)
    ref = H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), C.ADAM, state, ecc_bits, group)
    dev = ref.copy().to_device()
    g = H.make_grad(rng, n, 1e-2, np.float32)
    g[rng.integers(0, n, n // 100)] *= np.float32(1e22)
    hp = H.hyper_tuple(C.ADAM, conv, 1, lr=1e-3, wd=1e-2)
    H.oracle_step(C.ADAM, g, ref, state, group, hp)
    _step(C.ADAM, [H.to_torch(g)], [dev], None, state, group, hp, pdt, 0, ecc_bits)
    assert np.isfinite(ref.param.astype(np.float32)).all()
    H.assert_leaf_equal(dev.to_host(), ref, f"n={n}")


@pytest.mark.parametrize("n", [1000, MAIN + 700])
@pytest.mark.parametrize("opt,pdt,ecc_bits,group", [(C.ADAM, 2, 8, 16), (C.ADAM, 1, 16, 32), (C.LION, 2, 16, 128), (C.LION, 1, 8, 64), (C.SGD, 2, 8, 32)])
def test_parameters_that_are_infinite(opt, pdt, ecc_bits, group, n):
    """An infinity (an fp16 weight that left its range) stays one, with a code of zero, and its neighbours are stepped."""
    rng = np.random.default_rng(n)
    p = rng.normal(0, 0.02, n).astype(np.float32)
    p[rng.integers(0, n, n // 100)] = np.inf
    p[rng.integers(0, n, n // 100)] = -np.inf
    ref = H.fresh_leaf(p.astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, group)
    ref.ecc[:] = rng.integers(-100, 100, n)
    dev = ref.copy().to_device()
    g = H.make_grad(rng, n, 1e-2, H.BF16)
    hp = H.hyper_tuple(opt, O.FUSED, 1, lr=1e-3, wd=1e-2)
    H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
    _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, group, hp, pdt, 1, ecc_bits)
    H.assert_leaf_equal(dev.to_host(), ref, f"n={n}")


@pytest.mark.parametrize("n", [1000, MAIN + 700])
@pytest.mark.parametrize("opt,pdt,ecc_bits", [(C.ADAM, 1, 8), (C.ADAM, 2, 16), (C.LION, 1, 16), (C.SGD, 0, 0)])
def test_gradients_that_are_nan(opt, pdt, ecc_bits, n):
    """Their parameters become NaN and their codes 0; the scale of a group of 32 is that of its other elements, any other
    group's scale is NaN."""
    rng = np.random.default_rng(n)
    for group in (32, 128):
        ref = H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, group)
        dev = ref.copy().to_device()
        g = H.make_grad(rng, n, 1e-2, H.BF16)
        at = rng.integers(0, n, n // 100)
        g[at] = np.nan
        hp = H.hyper_tuple(opt, O.FUSED, 1, lr=1e-3, wd=1e-2)
        H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
        _step(opt, [H.to_torch(g)], [dev], None, C.STATE_QUANT, group, hp, pdt, 1, ecc_bits)
        got = dev.to_host()
        assert np.isnan(got.param[at].astype(np.float32)).all() and np.isnan(ref.param[at].astype(np.float32)).all()
        got.param[at] = ref.param[at]  # (whichever NaN it is)
        if group != 32:
            for name, codes in (("mu_scales", "mu"), ("nu_scales", "nu")):
                if getattr(ref, name) is not None:
                    hit = np.unique(at // group)
                    assert np.isnan(getattr(got, name)[hit]).all()
                    getattr(got, name)[hit] = getattr(ref, name)[hit]
                    inside = np.isin(np.arange(n) // group, hit)
                    getattr(got, codes)[inside] = getattr(ref, codes)[inside]  # of a group whose scale is NaN
        H.assert_leaf_equal(got, ref, f"n={n} group={group}")


@pytest.mark.parametrize("n", [1024, 20 * 1024 + 300, MAIN + 700])
@pytest.mark.parametrize("pdt,ecc_bits,group,conv,max_norm,elsewhere", [
    (1, 16, 32, O.FUSED, None, False), (2, 8, 32, O.FUSED, 0.5, False), (1, 8, 128, O.FUSED, None, False), (0, 0, 16, O.FUSED, 0.5, False),
    (1, 16, 32, O.UNFUSED, None, False), (1, 8, 32, O.FUSED, None, True)])
def test_rows_at_rest(pdt, ecc_bits, group, conv, max_norm, elsewhere, n):
    """AdamW on a leaf most of whose rows never see a gradient: only weight decay, in whole warps and in parts of them."""
    import torch

    from flashoptim_jax_b200 import _engine as eng

    rng = np.random.default_rng(n + group)
    ref = H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), C.ADAM, C.STATE_QUANT, ecc_bits, group)
    ref.param[600:700] = 0
    dev = ref.copy().to_device()
    for t in (1, 2):
        g = H.make_grad(rng, n, 1e-2, H.BF16)
        g[: n // 4] = 0
        g[n // 2 + 100 :] = -H.BF16.type(0)
        dev_g, sq, step_g = H.to_torch(g), None, g
        if max_norm is not None:
            sq = eng.sq_norm_of([dev_g])
            step_g = O.clip_by_global_norm([g], max_norm, sq_norm=float(sq.cpu()))[0]
        hp = H.hyper_tuple(C.ADAM, conv, t, lr=1e-3, wd=1e-2)
        H.oracle_step(C.ADAM, step_g, ref, C.STATE_QUANT, group, hp)
        outs = [H.LeafArrays(*[None if getattr(dev, f) is None else torch.empty_like(getattr(dev, f)) for f in dev.fields()])] if elsewhere else None
        _step(C.ADAM, [dev_g], [dev], outs, C.STATE_QUANT, group, hp, pdt, 1, ecc_bits, sq, max_norm or 0.0)
        dev = outs[0] if elsewhere else dev
        H.assert_leaf_equal(dev.to_host(), ref, f"step {t}")
    # codes of zero under an infinite scale are no rest: 0 * inf
    dev.mu_scales[:] = float("inf")
    dev.mu.zero_()
    ref.mu_scales[:] = np.inf
    ref.mu[:] = 0
    dev_g = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
    _step(C.ADAM, [dev_g], [dev], None, C.STATE_QUANT, group, hp, pdt, 1, ecc_bits)
    assert bool(torch.isnan(dev.param.float()).all())


@pytest.mark.parametrize("opt,group,conv,elsewhere", [(C.ADAM, 32, O.FUSED, False), (C.ADAM, 128, O.UNFUSED, False), (C.SGD, 40, O.FUSED, False),
                                                      (C.LION, 40, O.FUSED, True), (C.LION, 32, O.FUSED, True)])
def test_leaf_counts_around_the_table_sizes(opt, group, conv, elsewhere):
    """Kernel-parameter tables of 12, 236, 240 and 320 leaves, full, one over, and behind whole chunks."""
    for count in (12, 13, 236, 237, 240, 241, 320, 321, 700):
        _run(opt, 1, 8, C.STATE_QUANT, group, conv, [1 + i % 61 for i in range(count)], steps=1, elsewhere=elsewhere)
    _run(opt, 1, 8, C.STATE_QUANT, group, conv, [6000 + i for i in range(330)], steps=1, elsewhere=elsewhere)


@pytest.mark.parametrize("opt,pdt,ecc_bits,group,conv", [
    (C.ADAM, 1, 8, 32, O.FUSED), (C.ADAM, 2, 16, 32, O.FUSED), (C.ADAM, 0, 0, 64, O.FUSED), (C.ADAM, 1, 16, 32, O.UNFUSED),
    (C.LION, 1, 16, 32, O.FUSED), (C.LION, 1, 8, 32, O.UNFUSED), (C.SGD, 1, 8, 128, O.FUSED), (C.SGD, 2, 16, 32, O.FUSED)])
@pytest.mark.parametrize("elsewhere", [False, True])
def test_extreme_values_in_whole_chunks(opt, pdt, ecc_bits, group, conv, elsewhere):
    """Zeros, subnormals, huge and tiny values scattered and in whole groups through tile_kernel: nearly every warp takes the
    repairing pass."""
    import torch

    rng = np.random.default_rng(11)
    n = MAIN + 300
    p32 = np.ldexp(rng.normal(0, 1, n), np.clip(rng.integers(-140, 60, n), -140, 30)).astype(np.float32)
    p32[::7] = 0
    ref = H.fresh_leaf((np.clip(p32, -1e3, 1e3) if pdt == 2 else p32).astype(H.NP_OF_CODE[pdt]), opt, C.STATE_QUANT, ecc_bits, group)
    dev = ref.copy().to_device()
    for t in (1, 2):
        g = np.ldexp(rng.normal(0, 1, n), rng.integers(-140, 12, n)).astype(np.float32)
        g[::5] = 0
        g[5000:9000] = 0
        hp = H.hyper_tuple(opt, conv, t, lr=1e-3, wd=1e-2)
        H.oracle_step(opt, g, ref, C.STATE_QUANT, group, hp)
        outs = [H.LeafArrays(*[None if getattr(dev, f) is None else torch.empty_like(getattr(dev, f)) for f in dev.fields()])] if elsewhere else None
        _step(opt, [H.to_torch(g)], [dev], outs, C.STATE_QUANT, group, hp, pdt, 0, ecc_bits)
        dev = outs[0] if elsewhere else dev
        H.assert_leaf_equal(dev.to_host(), ref, f"step {t}")


@pytest.mark.parametrize("pdt,ecc_bits,state,group,max_norm", [(1, 8, C.STATE_QUANT, 32, None), (1, 16, C.STATE_QUANT, 128, 0.5), (2, 8, C.STATE_FULL, 32, None)])
@pytest.mark.parametrize("bc2", [0.5, 1e-12])
def test_device_scalars_in_whole_chunks(pdt, ecc_bits, state, group, max_norm, bc2):
    """Learning rate and bias corrections read from the device: a correction in the range of the reciprocal shortcut, and one outside it,
    which the kernel only sees once it runs (its tiles or chunks then go element by element)."""
    import torch

    from flashoptim_jax_b200 import _engine as eng

    rng = np.random.default_rng(5)
    n = MAIN + 77
    ref = H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.NP_OF_CODE[pdt]), C.ADAM, state, ecc_bits, group)
    dev = ref.copy().to_device()
    g = H.make_grad(rng, n, 1e-2, H.BF16)
    dev_g, sq, step_g = H.to_torch(g), None, g
    if max_norm is not None:
        sq = eng.sq_norm_of([dev_g])
        step_g = O.clip_by_global_norm([g], max_norm, sq_norm=float(sq.cpu()))[0]
    lr, bc1, bc2 = np.float32(2e-3), np.float32(0.25), np.float32(bc2)
    hp = list(H.hyper_tuple(C.ADAM, O.FUSED, 3, lr=lr, wd=1e-2))
    hp[7], hp[8] = bc1, bc2
    H.oracle_step(C.ADAM, step_g, ref, state, group, hp)
    scalars = torch.tensor([lr, bc1, bc2], device="cuda")
    host = list(H.hyper_tuple(C.ADAM, O.FUSED, 1, lr=0.5, wd=1e-2))  # what the host says about these three does not count
    H.abi_step(C.ADAM, [dev_g], [dev], state, group, [tuple(host) + (scalars.data_ptr(),)], [0], pdt, 1, ecc_bits, grad_sq_norm=sq,
               max_grad_norm=max_norm or 0.0)
    H.assert_leaf_equal(dev.to_host(), ref)


def test_nothing_is_written_beside_a_leaf_of_whole_chunks():
    """Guard bytes on both sides of every array of a leaf that ends inside a tile."""
    import torch

    rng = np.random.default_rng(2)
    n = MAIN + 333
    ref = H.fresh_leaf(rng.normal(0, 0.02, n).astype(np.float32).astype(H.BF16), C.ADAM, C.STATE_QUANT, 16)
    inner, framed = ref.copy().to_device(), {}
    for f in inner.fields():
        t = getattr(inner, f)
        framed[f] = torch.full((t.numel() * t.element_size() + 512,), 0xA5, dtype=torch.uint8, device="cuda")
        view = framed[f][256 : 256 + t.numel() * t.element_size()].view(t.dtype)
        view.copy_(t)
        setattr(inner, f, view)
    g = H.make_grad(rng, n, 1e-2, H.BF16)
    hp = H.hyper_tuple(C.ADAM, O.FUSED, 1, lr=1e-3, wd=1e-2)
    H.oracle_step(C.ADAM, g, ref, C.STATE_QUANT, 32, hp)
    _step(C.ADAM, [H.to_torch(g)], [inner], None, C.STATE_QUANT, 32, hp, 1, 1, 16)
    H.assert_leaf_equal(inner.to_host(), ref)
    for f, whole in framed.items():
        assert bool((whole[:256] == 0xA5).all()) and bool((whole[-256:] == 0xA5).all()), f
