"""Backward parity of `experts_backward` (through the C ABI) against autograd through the
reference's training branch (golden vectors) and against the CPU oracle."""
import pytest
import torch

from oracle import experts_oracle as orc
from helpers import RTOL_BF16, RTOL_F32, SMALL_CASES, backward_by_c_abi, golden_inputs, load_golden

pytestmark = pytest.mark.gpu
GRADS = ["d_hidden", "d_routing", "d_wgu", "d_bgu", "d_wd", "d_bd"]


def run_backward(grad_out, inp, capacity, E, K, path="auto"):
    import yamoe_b200
    yamoe_b200.set_path(path)
    try:
        outs = yamoe_b200.experts_backward(grad_out.cuda(), *[t.cuda() for t in inp], capacity, E, K)
        torch.cuda.synchronize()
    finally:
        yamoe_b200.set_path("auto")
    return [o.cpu() for o in outs]


@pytest.mark.parametrize("name", SMALL_CASES)
def test_backward_fp32_golden(name):
    g = load_golden(name)
    T, H, E, K = g["dims"].tolist()
    grads = run_backward(g["grad_out"], golden_inputs(g), T, E, K)
    for got, key in zip(grads, GRADS):
        orc.check_close(got, g[key], RTOL_F32, key)


@pytest.mark.parametrize("name", SMALL_CASES)
def test_backward_fp32_golden_dropping_capacity(name):
    """Against autograd through the reference's binned_experts_ref with a capacity that drops rows."""
    g, d = load_golden(name), load_golden("drop_grads")
    T, H, E, K = g["dims"].tolist()
    grads = run_backward(g["grad_out"], golden_inputs(g), int(d[f"{name}_cap"]), E, K)
    for got, key in zip(grads, GRADS):
        orc.check_close(got, d[f"{name}_{key}"], RTOL_F32, key + " (dropping capacity)")


def test_backward_capacity_drop_and_slot_shapes():
    g = load_golden("small_c")
    T, H, E, K = g["dims"].tolist()
    cap = int(g["cap_small"])
    inp = golden_inputs(g)
    ref = orc.experts_backward_oracle(g["grad_out"], *inp, cap, E, K)
    got = run_backward(g["grad_out"], inp, cap, E, K)
    for a, b, key in zip(got, ref, GRADS):
        orc.check_close(a, b, RTOL_F32, key + " (capacity drop)")
    # [T,K] routing weights and [T,K,H] grad_out
    inp_k = list(inp)
    inp_k[2] = torch.gather(g["routing_weights"], 1, g["router_indices"])
    gk = (g["grad_out"].unsqueeze(1).repeat(1, K, 1) / K).contiguous()
    ref = orc.experts_backward_oracle(gk, *inp_k, T, E, K)
    got = run_backward(gk, inp_k, T, E, K)
    assert got[1].shape == (T, K)
    for a, b, key in zip(got, ref, GRADS):
        orc.check_close(a, b, RTOL_F32, key + " (per-slot shapes)")


@pytest.mark.parametrize("path", ["simt", "auto"])
@pytest.mark.parametrize("T,H,E,K", [(96, 64, 4, 2), (512, 128, 8, 2), (1024, 256, 32, 4)])
def test_backward_bf16(path, T, H, E, K):
    inp = orc.make_inputs(T, H, E, K, seed=T + 1, weight_std=1.6 / (H ** 0.5), bias_std=0.2, dtype=torch.bfloat16,
                          with_grad=True)
    keys = ["hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
            "down_proj", "down_proj_bias"]
    args = [inp[k] for k in keys]
    ref = orc.experts_backward_oracle(inp["grad_out"], *args, T, E, K)
    got = run_backward(inp["grad_out"], args, T, E, K, path=path)
    for a, b, key in zip(got, ref, GRADS):
        assert a.dtype == torch.bfloat16
        orc.check_close(a.float(), b, RTOL_BF16, f"{key} bf16 ({path})", rel_l2=2e-2)


def test_autograd_function_end_to_end():
    import yamoe_b200
    g = load_golden("small_b")
    T, H, E, K = g["dims"].tolist()
    inp = [t.cuda() for t in golden_inputs(g)]
    for i in (0, 2, 3, 4, 5, 6):
        inp[i].requires_grad_(True)
    out = yamoe_b200.experts_autograd(*inp, T, E, K, True)
    (out * g["grad_out"].cuda()).sum().backward()
    orc.check_close(out.detach().cpu(), g["out_train"], RTOL_F32, "forward")
    for i, key in zip((0, 2, 3, 4, 5, 6), GRADS):
        orc.check_close(inp[i].grad.cpu(), g[key], RTOL_F32, key)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_saved_activation_pair_matches_recompute(dtype):
    """forward_saving + backward_saved give the output and gradients of experts + experts_backward."""
    import yamoe_b200
    T, H, E, K = 700, 256, 8, 2
    inp = orc.make_inputs(T, H, E, K, seed=21, weight_std=0.1, bias_std=0.2, dtype=dtype, with_grad=True)
    keys = ["hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
            "down_proj", "down_proj_bias"]
    for cap in (T, 120):
        dev = [inp[k].cuda() for k in keys]
        for i in (0, 2, 3, 4, 5, 6):
            dev[i].requires_grad_(True)
        out = yamoe_b200.experts_autograd(*dev, cap, E, K, True, save_activations=True)
        (out.float() * inp["grad_out"].cuda().float()).sum().backward()
        ref_out = orc.experts_forward_oracle(*[inp[k] for k in keys], cap, E, K)
        ref_g = orc.experts_backward_oracle(inp["grad_out"], *[inp[k] for k in keys], cap, E, K)
        tol = RTOL_F32 if dtype == torch.float32 else RTOL_BF16
        orc.check_close(out.detach().float().cpu(), ref_out, tol, f"saved-mode forward (capacity {cap})")
        for i, r, name in zip((0, 2, 3, 4, 5, 6), ref_g, GRADS):
            orc.check_close(dev[i].grad.float().cpu(), r, tol, f"saved-mode {name} (capacity {cap})",
                            rel_l2=None if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("T,H,E", [(130, 64, 3), (130, 128, 5), (130, 256, 4), (130, 320, 6), (130, 64, 150), (130, 128, 300),
                                   (600, 192, 2), (1100, 320, 3)])
def test_weight_gradients_of_few_rows(T, H, E):
    """Output rows and columns at the edges of the parked boxes, the bias row in a box of its own or behind others, experts
    without rows, more experts than leave space to park for four groups of warps, and enough rows for two groups."""
    K = 2
    inp = orc.make_inputs(T, H, E, K, seed=H + E, weight_std=H ** -0.5, bias_std=0.2, dtype=torch.bfloat16, with_grad=True)
    args = [inp[k] for k in ("hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
                             "down_proj", "down_proj_bias")]
    ref = orc.experts_backward_oracle(inp["grad_out"], *args, T, E, K)
    for a, b, key in zip(run_backward(inp["grad_out"], args, T, E, K), ref, GRADS):
        orc.check_close(a.float(), b, RTOL_BF16, key, rel_l2=2e-2)


@pytest.mark.parametrize("dense", [True, False])
@pytest.mark.parametrize("T,E,K,capacity", [(9, 40, 33, 4), (70, 70, 5, 3), (33, 8, 8, 100)])
def test_routing_gradient_of_every_column(T, E, K, capacity, dense):
    """d_routing is written whole: more slots than a warp has lanes, several rounds of columns, dropped assignments; nothing
    of it was set before (the allocator is made to hand out used memory)."""
    inp = orc.make_inputs(T, 64, E, K, seed=E + K, weight_std=0.125, bias_std=0.2, dtype=torch.float32, with_grad=True)
    args = [inp[k] for k in ("hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
                             "down_proj", "down_proj_bias")]
    if not dense:
        args[2] = torch.gather(args[2], 1, args[1]).contiguous()
    ref = orc.experts_backward_oracle(inp["grad_out"], *args, capacity, E, K)
    used = [torch.full((n,), float("nan"), device="cuda") for n in (T * E, T * K, T * 64) for _ in range(4)]
    del used
    for a, b, key in zip(run_backward(inp["grad_out"], args, capacity, E, K), ref, GRADS):
        orc.check_close(a, b, RTOL_F32, key)


@pytest.mark.parametrize("saved", [False, True])
@pytest.mark.parametrize("dtype,H,path,offset,accepted", [
    (torch.float32, 64, "auto", 2, True), (torch.float32, 64, "auto", 1, False), (torch.float32, 64, "simt", 2, False),
    (torch.float32, 72, "auto", 2, False), (torch.float32, 72, "auto", 4, True), (torch.bfloat16, 64, "auto", 4, True),
    (torch.bfloat16, 64, "auto", 2, False), (torch.bfloat16, 64, "simt", 4, True)])
def test_alignment_of_d_hidden(dtype, H, path, offset, accepted, saved):
    """In fp32 the sums of d_hidden are the caller's buffer.  What the kernels can address is served, the rest refused."""
    import yamoe_b200
    T, E, K = 130, 4, 2
    inp = orc.make_inputs(T, H, E, K, seed=H + offset, weight_std=H ** -0.5, bias_std=0.2, dtype=dtype, with_grad=True)
    args = [inp[k] for k in ("hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
                             "down_proj", "down_proj_bias")]
    yamoe_b200.set_path(path)
    try:
        status, got = backward_by_c_abi(inp["grad_out"], args, T, E, K, saved=saved, d_hidden_offset=offset)
    finally:
        yamoe_b200.set_path("auto")
    assert status == (0 if accepted else -1)
    if accepted:
        ref = orc.experts_backward_oracle(inp["grad_out"], *args, T, E, K)
        for a, b, key in zip(got, ref, GRADS):
            orc.check_close(a.float(), b, RTOL_F32 if dtype == torch.float32 else RTOL_BF16, key)


@pytest.mark.parametrize("saved", [False, True])
@pytest.mark.parametrize("T,E,K,capacity,dense", [(130, 4, 2, 37, True), (300, 16, 8, 90, False), (5, 8, 2, 1, True),
                                                  (700, 3, 2, 300, False)])
@pytest.mark.parametrize("dtype,H,path", [(torch.float32, 64, "auto"), (torch.float32, 72, "auto"), (torch.float32, 128, "simt"),
                                          (torch.bfloat16, 64, "auto"), (torch.bfloat16, 192, "auto"), (torch.bfloat16, 72, "auto")])
def test_dropped_rows_among_unset_memory(dtype, H, path, T, E, K, capacity, dense, saved):
    """A capacity that drops, on outputs and workspace full of NaN: every element of a gradient is written, and nothing that a
    kernel reads without having written it (padding behind the kept rows, rows of dropped assignments) reaches one."""
    import yamoe_b200
    inp = orc.make_inputs(T, H, E, K, seed=T + H, weight_std=H ** -0.5, bias_std=0.2, dtype=dtype, with_grad=True)
    args = [inp[k] for k in ("hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
                             "down_proj", "down_proj_bias")]
    if not dense:
        args[2] = torch.gather(args[2], 1, args[1]).contiguous()
    yamoe_b200.set_path(path)
    try:
        status, got = backward_by_c_abi(inp["grad_out"], args, capacity, E, K, saved=saved)
    finally:
        yamoe_b200.set_path("auto")
    assert status == 0
    ref = orc.experts_backward_oracle(inp["grad_out"], *args, capacity, E, K)
    for a, b, key in zip(got, ref, GRADS):
        orc.check_close(a.float(), b, RTOL_F32 if dtype == torch.float32 else RTOL_BF16, key)
