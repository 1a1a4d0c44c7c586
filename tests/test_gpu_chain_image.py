"""Inputs of dependent list ops that are prepared once for the whole grid and read by every CTA from a tagged image: every producer, from the
narrowest input that takes this way up, wide and narrow ones in turn (what a wider op left behind it in the image belongs to no later one),
run after run and in a replayed graph with other inputs: the bits of the same list with every input prepared by every CTA for itself, which at 512
threads are those of the kernels one by one."""
import pytest

from bonsai_b200 import synth

pytestmark = pytest.mark.gpu
EPS = 1e-6


PLAN = [(1024, 2048, "plain"), (2048, 7168, "norm"), (7168, 3072, "norm"), (3072, 17408, "norm"), (17408, 2048, "plain"), (2048, 9216, "plain"),
        (9216, 4096, "swiglu"), (4096, 17408, "norm"), (17408, 5120, "swiglu"), (5120, 1024, "norm"), (1024, 300, "norm")]


@pytest.mark.parametrize("threads", [512, 640, 768])
def test_widths_and_producers(gpu, threads):
    import torch
    to = lambda a: torch.from_numpy(a).cuda()
    xs = [to(synth.activations(1024, seed=s)) for s in range(3)]
    x0, scratch = xs[0].clone(), torch.zeros(17408 // 32 * 36, dtype=torch.uint8, device="cuda")
    flags = {"plain": 0, "norm": gpu.OP_RMSNORM, "swiglu": gpu.OP_SWIGLU}
    steps = [(to(synth.pq2_0_weights(n_out, n_in, seed=i)), to(synth.signs(n_in, seed=i)), to(synth.activations(n_in // 1024 * 1024, seed=40 + i)))
             for i, (n_in, n_out, _) in enumerate(PLAN)]

    def make(spread_nb):
        ys, ops = [torch.zeros(n_out, device="cuda") for _, n_out, _ in PLAN], []
        for i, ((n_in, n_out, kind), (W, sg, aux)) in enumerate(zip(PLAN, steps)):
            extra = {"plain": (), "norm": (aux, EPS), "swiglu": (aux,)}[kind]
            ops.append((W, ys[i - 1] if i else x0, sg, ys[i], n_out, n_in, flags[kind] | gpu.OP_ROTATE | (gpu.OP_DEPENDS if i else 0), *extra))
        try:
            assert gpu.set_option("chain_threads", threads) == 0 and gpu.set_option("chain_spread_nb", spread_nb) == 0
            return gpu.Chain(ops), ys
        finally:
            gpu.set_option("chain_threads", 512)
            gpu.set_option("chain_spread_nb", 16)

    def one_by_one():
        out, x = [], x0
        for (n_in, n_out, kind), (W, sg, aux) in zip(PLAN, steps):
            t, r = torch.empty(n_in, device="cuda"), torch.zeros(n_out, device="cuda")
            assert (gpu.rmsnorm(x, aux, t, 1, n_in, EPS) if kind == "norm" else gpu.swiglu(x, aux, t, n_in) if kind == "swiglu" else 0) == 0
            assert gpu.linear(W, x if kind == "plain" else t, sg, r, scratch, n_out, n_in) == 0
            out.append(r)
            x = r
        return out

    (chain, got), (other, want) = make(16), make(0)
    graph = torch.cuda.CUDAGraph()
    for run in range(6):
        x0.copy_(xs[run % 3])
        for y in got + want:
            y.fill_(-1.0)
        assert other.run() == 0
        if run == 3:
            with torch.cuda.graph(graph):
                assert chain.run() == 0
        if run < 3:
            assert chain.run() == 0
        else:
            graph.replay()
        torch.cuda.synchronize()
        assert gpu.device_status() == 0
        single = one_by_one() if threads == 512 else want
        for i in range(len(PLAN)):
            assert torch.equal(got[i], want[i]) and torch.equal(want[i], single[i]), (run, i)
    del graph
    chain.close()
    other.close()
