"""Shared helpers for the tests: golden loading and tolerance rules."""
import importlib
import os
import pickle

import numpy as np
import torch

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
SMALL_CASES = ["small_a", "small_b", "small_c", "small_d"]
INPUT_KEYS = ["hidden_states", "router_indices", "routing_weights", "gate_up_proj",
              "gate_up_proj_bias", "down_proj", "down_proj_bias"]

# Tolerances: |x - ref| <= rtol*|ref| + rtol*max|ref|, plus a rel-L2 bound for bf16.
RTOL_F32 = 1e-4
RTOL_BF16 = 2e-2
REL_L2_BF16 = 1e-2


class _Whole:
    """Arrives at the other end of a queue as the object that was put, tensors by value."""

    def __init__(self, obj):
        self.data = pickle.dumps(obj)

    def __reduce__(self):
        return pickle.loads, (self.data,)


class _WholeQueue:
    def __init__(self, queue):
        self.queue = queue

    def put(self, obj):
        self.queue.put(_Whole(obj))


def run_rank(module, worker, *args):
    """`worker` of a test module as a process, its queue (the last argument) passing tensors by value: by torch's own way a
    tensor goes as a file handle, which its reader has to fetch while the sending process still lives."""
    getattr(importlib.import_module(module), worker)(*args[:-1], _WholeQueue(args[-1]))


def load_golden(name):
    z = np.load(os.path.join(GOLDEN, name + ".npz"))
    return {k: torch.from_numpy(z[k]) if z[k].ndim else z[k].item() for k in z.files}


def backward_by_c_abi(grad_out, args, capacity, E, K, saved=False, d_hidden_offset=0):
    """yamoe_b200_experts_backward, or the saving pair, on buffers of the caller's: outputs and workspace hold NaN (and -1)
    before the call.  d_hidden starts `d_hidden_offset` elements behind a 16-byte boundary.  (status, gradients)"""
    from yamoe_b200 import _lib
    L = _lib.lib()

    def poisoned(nbytes):
        return torch.full((nbytes,), 0xFF, dtype=torch.uint8, device="cuda")

    dev = [t.cuda() for t in args]
    grad = grad_out.cuda()
    x, ridx, rw, wgu, bgu, wd, bd = [t.data_ptr() for t in dev]
    (T, H), cols, size = args[0].shape, args[2].shape[1], args[0].element_size()
    dtype = 0 if size == 4 else 1
    shapes = [t.shape for t in (args[0], args[2], *args[3:])]
    raw = [poisoned(s.numel() * size + 32) for s in shapes]
    lead = [d_hidden_offset * size] + [0] * 5
    grads = [r[o:o + s.numel() * size].view(args[0].dtype).view(s) for r, s, o in zip(raw, shapes, lead)]
    outs = [g.data_ptr() for g in grads]
    nbytes = L.yamoe_b200_backward_workspace_bytes(T, H, E, K, dtype)
    ws = poisoned(nbytes)
    assert ws.data_ptr() % 256 == 0 and all(r.data_ptr() % 16 == 0 for r in raw)
    tail = (T, H, E, K, capacity, dtype, ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)
    per_slot = int(grad_out.dim() == 3)
    if saved:
        out = poisoned(T * H * size)
        _lib.check(L.yamoe_b200_experts_forward_saving(x, ridx, rw, cols, wgu, bgu, wd, bd, out.data_ptr(), *tail), "saving forward")
        status = L.yamoe_b200_experts_backward_saved(grad.data_ptr(), per_slot, rw, cols, wgu, wd, bd, *outs, *tail)
    else:
        status = L.yamoe_b200_experts_backward(grad.data_ptr(), per_slot, x, ridx, rw, cols, wgu, bgu, wd, bd, *outs, *tail)
    torch.cuda.synchronize()
    return status, [g.cpu() for g in grads]


def golden_inputs(g):
    return [g[k] for k in INPUT_KEYS]
