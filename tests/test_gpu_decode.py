"""Decode-sized token counts: the weight-streaming GEMV path against the CPU oracle, and against
the grouped-GEMM path on the same inputs."""
import pytest
import torch

from oracle import experts_oracle as orc
from helpers import RTOL_BF16, REL_L2_BF16
from test_gpu_forward import run_experts

pytestmark = pytest.mark.gpu
KEYS = ["hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
        "down_proj", "down_proj_bias"]


@pytest.mark.parametrize("T", [1, 4, 16, 64])
def test_decode_gemv_120b_like(T):
    H, E, K = 512, 128, 4
    inp = orc.make_inputs(T, H, E, K, seed=42 + T, weight_std=0.05, bias_std=0.1, dtype=torch.bfloat16)
    args = [inp[k] for k in KEYS]
    ref = orc.experts_forward_oracle(*args, T, E, K)
    out = run_experts(args, T, E, K, path="gemv")
    orc.check_close(out.float(), ref, RTOL_BF16, f"gemv T={T}", rel_l2=REL_L2_BF16)
    auto = run_experts(args, T, E, K, path="auto")          # auto picks the GEMV path here
    assert torch.equal(auto, out) or (auto.float() - out.float()).abs().max() <= 2e-2 * ref.abs().max()


@pytest.mark.parametrize("T,H,E,K,cap", [(3, 64, 5, 2, 3), (7, 136, 4, 1, 2), (40, 64, 2, 2, 64), (9, 2880, 6, 3, 9),
                                          (128, 64, 8, 2, 128), (32, 64, 1, 1, 32)])
def test_decode_gemv_shapes_and_capacity(T, H, E, K, cap):
    inp = orc.make_inputs(T, H, E, K, seed=T * 7 + H, weight_std=1.0 / (H ** 0.5), bias_std=0.2,
                          dtype=torch.bfloat16)
    args = [inp[k] for k in KEYS]
    ref = orc.experts_forward_oracle(*args, cap, E, K)
    out = run_experts(args, cap, E, K, path="gemv")
    orc.check_close(out.float(), ref, RTOL_BF16, "gemv", rel_l2=REL_L2_BF16)


def test_decode_gemv_topk_weights():
    T, H, E, K = 5, 64, 16, 4
    inp = orc.make_inputs(T, H, E, K, seed=3, weight_std=0.1, bias_std=0.2, dtype=torch.bfloat16)
    args = [inp[k] for k in KEYS]
    ref = orc.experts_forward_oracle(*args, T, E, K)
    args[2] = torch.gather(inp["routing_weights"], 1, inp["router_indices"])
    out = run_experts(args, T, E, K, path="gemv")
    orc.check_close(out.float(), ref, RTOL_BF16, "gemv per-slot weights", rel_l2=REL_L2_BF16)


@pytest.mark.parametrize("T,H,E,K", [(16, 2880, 128, 4), (32, 2880, 128, 4), (16, 2880, 32, 4), (32, 2880, 32, 4),
                                     (16, 2048, 64, 8), (32, 2048, 64, 8), (31, 1024, 32, 4), (43, 2048, 64, 3)])
def test_decode_rows_are_summed_in_fp32(T, H, E, K):
    """Whichever kernels `auto` picks for a decode-sized call, no result is rounded to bf16 more often than on the
    weight-streaming path: activations and output, not the K rows of a token.  Then the errors against 64 bits
    agree but for elements whose fp32 sums fall on different sides of a rounding boundary (a row
    rounding raises the error by a fifth)."""
    inp = orc.make_inputs(T, H, E, K, seed=T + E, weight_std=0.02, bias_std=0.02, dtype=torch.bfloat16, weights_on="cuda")
    args = [inp[k] for k in KEYS]
    ref = orc.experts_forward_oracle(*[a.cpu() for a in args], T, E, K, compute_dtype=torch.float64)
    gemv, auto = run_experts(args, T, E, K, path="gemv"), run_experts(args, T, E, K, path="auto")
    err = [((o.double() - ref).norm() / ref.norm()).item() for o in (gemv, auto)]
    assert err[1] <= 1.02 * err[0], err
