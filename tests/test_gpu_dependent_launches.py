"""Launches start before the kernel in front of them has drained and wait inside: results of a chain of dependent calls on one
stream, each the next one's input and mixed with torch's kernels, equal those of the same calls with the device idle between them."""

import pytest

pytestmark = pytest.mark.gpu


def _chain(name, n, pause):
    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import clipping

    g = torch.Generator(device="cuda").manual_seed(n)
    p = {"w": (torch.randn(n, device="cuda", generator=g) * 0.02).bfloat16(), "b": torch.ones(33, device="cuda"), "c": torch.ones(5, device="cuda", dtype=torch.float16)}
    noise = torch.randn(n, device="cuda", generator=g) * 1e-3
    tx = clipping.clip_by_global_norm(getattr(fo, name)(learning_rate=1e-2, donate=True), 0.5)
    s = tx.init(p)
    pause()
    for _ in range(6):
        # the gradients are made from the parameters the step in front has just written
        grads = {"w": (p["w"].float() + noise).bfloat16(), "b": p["b"] * 0.1, "c": p["c"] * 0.5}
        pause()
        p, s = tx.step(p, s, grads)
        pause()
        w = fo.reconstruct_weights(p, s["opt"].ecc)
        pause()
        q = fo.quantize_momentum(w["w"], 32)
        pause()
        noise = fo.dequantize_momentum(q, 32)  # read by the next gradients
        pause()
        lp, ecc = fo.set_fp32_params(w, p, master_weight_bits=24)
        pause()
        p["w"].copy_(lp["w"])
        pause()
    return p, s, noise, q


@pytest.mark.parametrize("name", ["flash_adamw", "flash_lion", "flash_sgdw"])
@pytest.mark.parametrize("n", [1000, 2_000_003])  # pieces only; whole chunks and a ragged end
def test_dependent_calls_see_each_other(name, n):
    import torch

    from flashoptim_jax_b200 import tree

    a = tree.tree_leaves(_chain(name, n, lambda: None))
    torch.cuda.synchronize()
    b = tree.tree_leaves(_chain(name, n, torch.cuda.synchronize))
    for x, y in zip(a, b):
        assert torch.equal(x, y)


@pytest.mark.parametrize("name", ["flash_adamw", "flash_lion", "flash_sgdw"])
@pytest.mark.parametrize("n", [1000, 700_001, 2_000_003])
def test_launches_of_one_step_in_a_graph(name, n):
    """Leaves of three dtypes, the small ones first in the tree: their launches do not wait for that of the large one, the next gradients wait for all."""
    import torch

    import flashoptim_jax_b200 as fo
    from flashoptim_jax_b200 import tree

    def start():
        g = torch.Generator(device="cuda").manual_seed(n)
        p = {"a": torch.ones(4133, device="cuda"), "b": torch.ones(5, device="cuda", dtype=torch.float16),
             "w": (torch.randn(n, device="cuda", generator=g) * 0.02).bfloat16()}
        tx = getattr(fo, name)(learning_rate=1e-2, donate=True, capturable=True)
        return tx, p, tx.init(p)

    def steps(tx, p, s, pause):
        for _ in range(3):
            grads = {k: (v.float() * 0.1 + 1e-3).to(v.dtype) for k, v in p.items()}
            pause()
            p, s = tx.step(p, s, grads)
            pause()
        return p, s

    side = torch.cuda.Stream()
    tx, p, s = start()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        p, s = steps(tx, p, s, lambda: None)
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p, s = steps(tx, p, s, lambda: None)
    graph.replay()
    graph.replay()
    tx, q, t = start()
    for _ in range(3):
        q, t = steps(tx, q, t, torch.cuda.synchronize)
    torch.cuda.synchronize()
    for x, y in zip(tree.tree_leaves((p, s)), tree.tree_leaves((q, t))):
        assert torch.equal(x, y)
