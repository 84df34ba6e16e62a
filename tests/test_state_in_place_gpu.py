"""A lean backward through the C ABI whose gradient of the initial state takes the place of the state: the scan that still reads
the state does not run beside the one that writes the gradient."""

import ctypes as C

import pytest
import torch

from delta_feedback_experiment_b200 import _lib, ops
from delta_feedback_experiment_b200.synthetic import INPUT_NAMES, make_inputs
from test_launch_order_gpu import captured_launches

pytestmark = pytest.mark.gpu
D = 128
SAVED = ("Aqk", "Akk", "k_precond", "ac_atk", "a_atk", "sa_atk", "w", "kg", "v_new", "h", "qg")
GRADS = ("dq", "dk", "dv", "dg", "dg_atk", "dbeta_atk", "dbeta", "dA_log", "ddt_bias", "dlog_atk_scale")
OF = dict(zip(GRADS, ("q", "k", "v", "g", "g_atk", "beta_atk", "beta", "A_log", "dt_bias", "log_atk_scale")))


def _call(d, dS, states, shift):
    """Arguments of a lean backward and the tensors behind them.  ``states`` holds the initial state at its start and takes the
    gradient ``shift`` floats further on."""
    B, T, H, _ = d["q"].shape
    n = B * H * D * D
    S0, dS0 = (states[at:at + n].view(B, H, D, D) for at in (0, shift))
    S0.copy_(d["initial_state"])
    saved = ops.chunk_forward(*(d[x] for x in INPUT_NAMES), D ** -0.5, 1.5, 1e-6, S0, d["initial_A_state"])[3]
    out = {g: torch.empty_like(d[x]) for g, x in OF.items()}
    out.update(d_initial_state=dS0, d_initial_A_state=torch.empty_like(d["initial_A_state"]))
    a = _lib.ChunkBwdArgs()
    p = a.p
    p.n_seqs, p.seq_len, p.total_tokens, p.heads, p.head_dim, p.dtype = B, T, B * T, H, D, _lib.PKDA_BF16
    p.scale, p.squash_x, p.squash_eps = D ** -0.5, 1.5, 1e-6
    for x in INPUT_NAMES:
        setattr(p, x, d[x].data_ptr())
    p.initial_state, p.initial_A_state = S0.data_ptr(), d["initial_A_state"].data_ptr()
    a.d_o, a.d_final_state, a.recompute = d["do"].data_ptr(), dS.data_ptr(), 1
    for name, t in [*zip(SAVED, saved), *out.items()]:
        setattr(a, name, t.data_ptr())
    need = _lib.load().pkda_chunk_bwd_workspace_bytes(C.byref(p))
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), need
    return a, out, (saved, ws, states)


def _backward(a):
    assert _lib.load().pkda_chunk_bwd(C.byref(a), _lib.current_stream()) == 0


# 4, 16 and 36 units by columns, 40 by the tensor-memory scans; the gradient in the state's place, one unit behind it, and apart
@pytest.mark.parametrize("B,H", [(1, 4), (2, 8), (3, 12), (4, 10)])
def test_gradient_of_the_state_in_the_states_place(B, H):
    d = make_inputs(B, 200, H, D, seed=B, dist="production", dtype=torch.bfloat16, with_state=True)
    d = {n: t.cuda().contiguous() for n, t in d.items() if torch.is_tensor(t)}
    dS = torch.randn(B, H, D, D, device="cuda") * 0.1
    n, want = B * H * D * D, None
    for shift in (n, 0, D * D):
        states = torch.zeros(2 * n, device="cuda")
        a, out, keep = _call(d, dS, states, shift)
        _backward(a)
        torch.cuda.synchronize()
        got = {name: t.clone() for name, t in out.items()}
        if want is None:
            want = got
        for name in want:
            assert torch.equal(got[name], want[name]), (shift, name)
        del keep


def test_scans_of_overlapping_states_run_alone():
    """16 units: four CTAs a unit for each scan side by side, eight where a scan runs alone."""
    B, H = 2, 8
    d = make_inputs(B, 200, H, D, seed=3, dist="production", dtype=torch.bfloat16, with_state=True)
    d = {n: t.cuda().contiguous() for n, t in d.items() if torch.is_tensor(t)}
    dS = torch.randn(B, H, D, D, device="cuda") * 0.1
    n = B * H * D * D
    for shift, grid in ((n, 64), (0, 128), (n - 4, 128)):
        a, _, keep = _call(d, dS, torch.zeros(2 * n, device="cuda"), shift)
        _backward(a)
        torch.cuda.synchronize()
        scans = [x.grid for x in captured_launches(lambda: _backward(a)) if "pkda_scan_" in x.name]
        assert scans == [grid, grid], shift
        del keep
