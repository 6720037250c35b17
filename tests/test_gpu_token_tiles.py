"""The grouped GEMMs at the numbers of rows per expert where a tile or a k-block ends, the routing of many
assignments, and special values in fp32: against the CPU oracle, with the tolerances of the other tests."""
import pytest
import torch

from oracle import experts_oracle as orc
from helpers import REL_L2_BF16, RTOL_BF16, RTOL_F32

pytestmark = pytest.mark.gpu
GRADS = ["d_hidden", "d_routing", "d_wgu", "d_bgu", "d_wd", "d_bd"]
#: rows per expert: none, around the 16-row step, a 64-deep k-block, the 96 / 128 / 256-row boxes and tiles
COUNTS = [0, 1, 15, 16, 17, 63, 64, 65, 97, 129, 193, 255, 256, 257, 300, 513]


def _problem(counts, H, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    E, T = len(counts), sum(counts)
    ridx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(T, generator=g)][:, None]

    def normal(*shape, std):
        return (torch.randn(*shape, generator=g) * std).to(dtype)

    # Pre-activations of standard deviation 1: the clamp at 7 is never within rounding.  (A bf16
    # pre-activation that rounds to the other side of it switches its gradient on or off, an error of
    # the gradient's own size that no rounding bound covers: seen with a standard deviation of 1.8.)
    args = [normal(T, H, std=1.0), ridx, torch.rand(T, 1, generator=g).to(dtype) + 0.25,
            normal(E, H, 2 * H, std=H ** -0.5), normal(E, 2 * H, std=0.2), normal(E, H, H, std=H ** -0.5),
            normal(E, H, std=0.2)]
    return args, normal(T, H, std=1.0), T, E


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("H", [64, 192, 320])
@pytest.mark.parametrize("capacity", [10000, 130])
def test_rows_per_expert_at_tile_edges(dtype, H, capacity):
    import yamoe_b200
    from yamoe_b200.layers import experts_autograd
    args, grad, T, E = _problem(COUNTS, H, dtype, seed=H + capacity)
    rtol, l2 = (RTOL_BF16, REL_L2_BF16) if dtype == torch.bfloat16 else (RTOL_F32, RTOL_F32)
    dev = [a.cuda() for a in args]
    ref = orc.experts_forward_oracle(*args, capacity, E, 1)
    orc.check_close(yamoe_b200.experts(*dev, capacity, E, 1).float().cpu(), ref, rtol, "forward", rel_l2=l2)
    ref_g = orc.experts_backward_oracle(grad, *args, capacity, E, 1)
    got = yamoe_b200.experts_backward(grad.cuda(), *dev, capacity, E, 1)
    for a, b, n in zip(got, ref_g, GRADS):
        orc.check_close(a.float().cpu(), b, rtol, n)
    leaves = [t.requires_grad_(True) for t in dev if t.is_floating_point()]
    out = experts_autograd(*dev, capacity, E, 1, save_activations=True)
    orc.check_close(out.detach().float().cpu(), ref, rtol, "saving forward", rel_l2=l2)
    for a, i in zip(torch.autograd.grad(out, leaves, grad.cuda()), [0, 1, 2, 3, 4, 5]):
        orc.check_close(a.float().cpu(), ref_g[i], rtol, GRADS[i] + " (saved activations)")


@pytest.mark.parametrize("first,second", [("auto", "simt"), ("simt", "auto")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
def test_saved_activations_survive_a_change_of_path(first, second, dtype):
    """The buffer of the saving forward is consumed by the kernels of another path."""
    import yamoe_b200
    from yamoe_b200.layers import experts_autograd
    args, grad, T, E = _problem([0, 5, 70, 130], 64, dtype, seed=3)
    torch.full((1 << 24,), float("nan"), device="cuda")          # what the allocator hands out next is not zero
    dev = [a.cuda() for a in args]
    leaves = [t.requires_grad_(True) for t in dev if t.is_floating_point()]
    try:
        yamoe_b200.set_path(first)
        out = experts_autograd(*dev, T, E, 1, save_activations=True)
        yamoe_b200.set_path(second)
        got = torch.autograd.grad(out, leaves, grad.cuda())
    finally:
        yamoe_b200.set_path("auto")
    ref = orc.experts_backward_oracle(grad, *args, T, E, 1)
    for a, b, n in zip(got, ref, GRADS):
        orc.check_close(a.float().cpu(), b, RTOL_BF16 if dtype == torch.bfloat16 else RTOL_F32, n)


def _moved(t, floats):
    """A contiguous copy that starts `floats` elements behind a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device="cuda")
    assert buf.data_ptr() % 16 == 0
    return buf[floats:floats + t.numel()].view(t.shape).copy_(t)


@pytest.mark.parametrize("H", [64, 192])
@pytest.mark.parametrize("forward,backward", [(1, 0), (0, 1), (1, 1), (0, 0)])
def test_saved_activations_survive_weights_that_move(H, forward, backward):
    """fp32 weights at 4-byte alignment run on the CUDA cores, aligned ones on the tensor cores: the saved buffer
    does not depend on which, so the weights may lie elsewhere in the backward pass."""
    import yamoe_b200
    args, grad, T, E = _problem([0, 5, 70, 130], H, torch.float32, seed=3)
    dev = [a.cuda() for a in args]
    out, saved = yamoe_b200.ops.experts_forward_saving(*dev[:3], _moved(dev[3], forward), dev[4],
                                                       _moved(dev[5], forward), dev[6], T, E, 1)
    got = yamoe_b200.ops.experts_backward_saved(grad.cuda(), saved, dev[2], _moved(dev[3], backward),
                                                _moved(dev[5], backward), dev[6], T, E, 1)
    orc.check_close(out.cpu(), orc.experts_forward_oracle(*args, T, E, 1), RTOL_F32, "saving forward")
    for a, b, n in zip(got, orc.experts_backward_oracle(grad, *args, T, E, 1), GRADS):
        orc.check_close(a.cpu(), b, RTOL_F32, n)


@pytest.mark.parametrize("path", ["simt", "auto"])
def test_saving_forward_runs_on_the_selected_path(path):
    """K = 1: one product sum per output, so that the same kernels give the same bits."""
    import yamoe_b200
    args, grad, T, E = _problem([0, 5, 70, 130], 192, torch.float32, seed=4)
    dev = [a.cuda() for a in args]
    yamoe_b200.set_path(path)
    try:
        plain, (out, saved) = yamoe_b200.experts(*dev, T, E, 1), yamoe_b200.ops.experts_forward_saving(*dev, T, E, 1)
        got = yamoe_b200.ops.experts_backward_saved(grad.cuda(), saved, dev[2], dev[3], dev[5], dev[6], T, E, 1)
        ref = yamoe_b200.experts_backward(grad.cuda(), *dev, T, E, 1)
    finally:
        yamoe_b200.set_path("auto")
    assert torch.equal(out, plain)
    for i in (2, 3, 4, 5):                    # the other two are sums of atomics
        assert torch.equal(got[i], ref[i]), GRADS[i]


@pytest.mark.parametrize("T,E,K", [(8193, 7, 4), (8191, 300, 4), (9001, 16, 4), (2731, 33, 3)])
def test_routing_of_many_assignments(T, E, K):
    """Around 32768 assignments, with ids outside [0, E) and a capacity that drops."""
    import yamoe_b200
    H = 64
    g = torch.Generator().manual_seed(T)
    ridx = torch.stack([torch.randperm(E, generator=g)[:K] for _ in range(64)]).repeat((T + 63) // 64, 1)[:T]
    ridx[5, 0], ridx[T - 1, K - 1] = -3, E + 2
    rw = torch.rand(T, K, generator=g)
    args = [torch.randn(T, H, generator=g), ridx, rw] + [torch.randn(*s, generator=g) * 0.1 for s in
                                                         ((E, H, 2 * H), (E, 2 * H), (E, H, H), (E, H))]
    cap = max(1, T * K // E - 3)
    # an id out of range contributes nothing: the oracle gets expert 0 with weight zero, behind everybody else
    rank = torch.zeros_like(ridx)
    seen = torch.zeros(E, dtype=torch.long)
    for p, e in enumerate(ridx.reshape(-1).tolist()):
        if 0 <= e < E:
            rank.view(-1)[p] = seen[e]
            seen[e] += 1
    keep = (rank < cap) & (ridx >= 0) & (ridx < E)
    w = torch.where(keep, rw, torch.zeros_like(rw))
    ref = orc.experts_forward_oracle(args[0], ridx.clamp(0, E - 1), w, *args[3:], T * K, E, K)
    out = yamoe_b200.experts(*[a.cuda() for a in args], cap, E, K)
    orc.check_close(out.cpu(), ref, RTOL_F32, "forward")


def test_fp32_products_keep_24_bits():
    """One token: the gate_up weight gradient is a single product x_i * g_j, the bias gradient g_j itself (x = 1).
    The bf16 parts that are multiplied leave out at most 2^-24 of a product, and the accumulator is cut off
    once at its full magnitude (2^-23) and five times at 2^-7 of it or less."""
    import yamoe_b200
    H, g = 64, torch.Generator().manual_seed(8)
    worst = [0x3f80ffff, 0x3f817fff, 0x3f807fff, 0x3f80ff7f, 0x3f8080ff, 0x3fffffff, 0x3f7fffff, 0x3f808080]
    bits = torch.tensor(worst * 4 + [0] * 32, dtype=torch.int32)
    x = torch.where(bits != 0, bits.view(torch.float32), torch.randn(H, generator=g))
    x = (x * 2.0 ** torch.randint(-9, 3, (H,), generator=g) * (1 - 2 * torch.randint(0, 2, (H,), generator=g))).view(1, H)
    args = [x, torch.zeros(1, 1, dtype=torch.long), torch.ones(1, 1)] + [
        torch.randn(*s, generator=g) * 0.1 for s in ((1, H, 2 * H), (1, 2 * H), (1, H, H), (1, H))]
    grads = yamoe_b200.experts_backward(torch.randn(1, H, generator=g).cuda(), *[a.cuda() for a in args], 1, 1, 1)
    got, bias = grads[2][0].cpu().double(), grads[3][0].cpu().double()
    want = x[0].double()[:, None] * bias[None, :]
    assert (want != 0).all()
    assert ((got - want) / want).abs().max().item() <= 2.0 ** -24 + 2.0 ** -23 + 5 * 2.0 ** -30


@pytest.mark.parametrize("H", [64, 320, 1024])
def test_fp32_against_64_bits(H):
    """Relative error in the 2-norm.  A GEMM's 64-deep blocks are cut off about four times at full magnitude
    (4 * 2^-23) and their sums rounded; a forward is two of them and the activation's few units of 2^-23, a
    gradient one more: 16 * 2^-23.  Without the third parts of the operands it is about 1e-5."""
    import yamoe_b200
    args, grad, T, E = _problem([0, 5, 70, 130, 33], H, torch.float32, seed=9)
    dev = [a.cuda() for a in args]
    got = [yamoe_b200.experts(*dev, T, E, 1), *yamoe_b200.experts_backward(grad.cuda(), *dev, T, E, 1)]
    ref = [orc.experts_forward_oracle(*args, T, E, 1, compute_dtype=torch.float64),
           *orc.experts_backward_oracle(grad, *args, T, E, 1, compute_dtype=torch.float64)]
    for a, b, n in zip(got, ref, ["out"] + GRADS):
        assert ((a.cpu().double() - b).norm() / b.norm()).item() <= 16 * 2.0 ** -23, n


@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.0e38, 3.395e38])
def test_fp32_parts_of_special_values(value):
    """Every output is NaN, infinite or finite where the CUDA-core kernel's is; weights are multiples of
    1/64, whose lower parts vanish.  bf16 rounds 3.395e38 to infinity."""
    import yamoe_b200
    args, grad, T, E = _problem([20, 33, 0, 70], 128, torch.float32, seed=5)
    for i in (3, 5):
        args[i] = (args[i] * 64).round() / 64
    args[0][7, 3], args[3][1, 5, 11], args[5][3, 9, 2] = value, value, -value
    dev = [a.cuda() for a in args]
    res = {}
    for path in ("auto", "simt"):
        yamoe_b200.set_path(path)
        try:
            res[path] = [yamoe_b200.experts(*dev, T, E, 1), *yamoe_b200.experts_backward(grad.cuda(), *dev, T, E, 1)]
            out, saved = yamoe_b200.ops.experts_forward_saving(*dev, T, E, 1)
            res[path] += [out, *yamoe_b200.ops.experts_backward_saved(grad.cuda(), saved, dev[2], dev[3], dev[5], dev[6],
                                                                      T, E, 1)]
        finally:
            yamoe_b200.set_path("auto")
    for a, b in zip(res["auto"], res["simt"]):
        assert torch.equal(a.isnan(), b.isnan())
        assert torch.equal(a.isinf() & (a > 0), b.isinf() & (b > 0)) and torch.equal(a.isinf(), b.isinf())


@pytest.mark.parametrize("counts", [[79, 80, 81, 0, 95, 97], [112, 113, 127, 129, 144], [145, 159, 160, 161], [320, 321, 1, 480],
                                    [1] * 400 + [0] * 500 + [161, 33]], ids=["80", "128", "160", "320", "many experts"])
def test_fp32_tile_sizes(counts):
    """Rows around the tile sizes that the fp32 kernel chooses from, and more experts than leave room for four stages."""
    import yamoe_b200
    args, grad, T, E = _problem(counts, 64, torch.float32, seed=len(counts))
    dev = [a.cuda() for a in args]
    ref = orc.experts_forward_oracle(*args, T, E, 1)
    orc.check_close(yamoe_b200.experts(*dev, T, E, 1).cpu(), ref, RTOL_F32, "forward")
    ref_g = orc.experts_backward_oracle(grad, *args, T, E, 1)
    for a, b, n in zip(yamoe_b200.experts_backward(grad.cuda(), *dev, T, E, 1), ref_g, GRADS):
        orc.check_close(a.cpu(), b, RTOL_F32, n)
