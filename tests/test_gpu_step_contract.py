"""What lbk_step_run takes beside what the models give it: caches whose layers lie apart by more than they hold. Equality with the bits of the plain call:
the same kernel on the same values."""
import pytest

pytestmark = pytest.mark.gpu


def _model(ctx, hidden, inner, heads, kv, layers, most):
    from lemonade_burn_b200 import model
    cfg = model.Config(hidden, inner, heads, kv, layers, 500, 1e-5, 500000.0, most)
    return model.BitNet(cfg, model.random_checkpoint(cfg, hidden + layers, "cuda"), ctx)


class Run:
    """A cache of random rows with `gap` elements more a layer than it holds, and steps on it from position `start`."""

    def __init__(self, net, b, cap, start, work, gap=0, seed=1):
        import torch
        self.net, self.b, self.cap, self.work = net, b, cap, work
        self.each = b * net.cfg.num_key_value_heads * cap * 128
        self.stride = self.each + gap
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        rows = torch.randn(2, net.cfg.num_hidden_layers, self.each, generator=self.gen, device="cuda").to(torch.bfloat16)
        n = net.cfg.num_hidden_layers * self.stride
        self.kv = torch.zeros(2, n + -n % 8, dtype=torch.bfloat16, device="cuda")  # both on 16 bytes
        self.layers()[:] = rows
        self.pos = torch.full((b,), start, dtype=torch.int32, device="cuda")

    def layers(self):
        return self.kv[:, :self.net.cfg.num_hidden_layers * self.stride].view(2, -1, self.stride)[:, :, :self.each]

    def step(self):
        import torch
        from lemonade_burn_b200 import _lib
        x = torch.randn(self.b, self.net.cfg.hidden_size, generator=self.gen, device="cuda")
        out = torch.empty_like(x)
        _lib.check(_lib.load().lbk_step_run(self.net._step.handle, self.b, self.cap, x.data_ptr(), self.kv[0].data_ptr(), self.kv[1].data_ptr(), self.stride,
                                            self.net.cos.data_ptr(), self.net.sin.data_ptr(), self.pos.data_ptr(), 1, self.work.data_ptr(), out.data_ptr(),
                                            torch.cuda.current_stream().cuda_stream))
        self.pos += 1
        return out


def _work(net, b, cap):
    import torch
    return torch.zeros(net._step.work_bytes(b, cap), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("b", [1, 3])
@pytest.mark.parametrize("gap", [4, 12, 8, 128])
def test_layers_that_lie_apart(ctx, gap, b):
    """Any multiple of four elements from layer to layer, those that leave every other layer on 8 bytes included."""
    import torch
    net, cap = _model(ctx, 512, 768, 4, 1, 3, 300), 300
    plain, apart = (Run(net, b, cap, 250, _work(net, b, cap), g) for g in (0, gap))
    assert plain.kv[1].data_ptr() % 16 == 0 and apart.kv[1].data_ptr() % 16 == 0
    for _ in range(3):
        assert torch.equal(plain.step(), apart.step())
    assert torch.equal(plain.layers(), apart.layers())
    ctx.check_device_error()


def test_one_buffer_for_launches_of_any_size(ctx):
    """A work buffer serves launches that come one after another whatever their sizes: other capacities (other slices of the positions), another
    model, several sequences in between, and back. With one sequence a value in the buffer says by itself that it is there, so what a launch of other
    sizes left must not be taken for it."""
    import torch
    nets = [_model(ctx, 512, 768, 4, 1, 3, 2000), _model(ctx, 1280, 3408, 10, 5, 2, 700)]
    sizes = [(0, 1, 2000), (0, 1, 70), (0, 3, 300), (1, 1, 700), (0, 16, 64), (1, 2, 128), (0, 1, 640)]
    shared = torch.zeros(max(nets[n]._step.work_bytes(b, cap) for n, b, cap in sizes), dtype=torch.uint8, device="cuda")
    own = [Run(nets[n], b, cap, cap - 40, _work(nets[n], b, cap), seed=cap + b) for n, b, cap in sizes]
    one = [Run(nets[n], b, cap, cap - 40, shared, seed=cap + b) for n, b, cap in sizes]
    order = [0, 1, 0, 2, 0, 3, 0, 4, 1, 5, 3, 6, 0, 6, 1, 3, 2, 4, 2, 0, 0, 1, 1, 5, 4, 3, 3, 0]
    got = [one[i].step() for i in order]
    torch.cuda.synchronize()
    want = [own[i].step() for i in order]
    for i, (g, w) in enumerate(zip(got, want)):
        assert torch.isfinite(w).all() and torch.equal(g, w), (i, sizes[order[i]])
    for a, b in zip(one, own):
        assert torch.equal(a.kv, b.kv)
    ctx.check_device_error()


def test_buffer_in_front_of_a_captured_step(ctx):
    """A graph that holds a step replays soundly behind launches of other sizes on its buffer."""
    import torch
    net = _model(ctx, 512, 768, 4, 1, 3, 2000)
    work = _work(net, 3, 2000)
    a, ref = (Run(net, 1, 2000, 1000, w, seed=3) for w in (work, _work(net, 1, 2000)))
    other = Run(net, 3, 2000, 500, work, seed=4)
    x = torch.randn(1, 512, device="cuda")

    def call(run, out):
        from lemonade_burn_b200 import _lib
        _lib.check(_lib.load().lbk_step_run(net._step.handle, 1, 2000, x.data_ptr(), run.kv[0].data_ptr(), run.kv[1].data_ptr(), run.stride, net.cos.data_ptr(),
                                            net.sin.data_ptr(), run.pos.data_ptr(), 1, run.work.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream))

    got, want, graph = torch.empty_like(x), torch.empty_like(x), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        call(a, got)
    for _ in range(4):
        other.step()
        graph.replay()
        call(ref, want)
        assert torch.equal(got, want)
        a.pos += 1
        ref.pos += 1
    ctx.check_device_error()
