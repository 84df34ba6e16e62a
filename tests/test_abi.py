"""CPU checks of the C-ABI boundary: the library loads, exports every symbol the
header declares, its struct layouts match the ctypes mirror, and argument
validation answers with status codes (no kernel is launched here)."""

import ctypes as C
import os
import re

import pytest

from conftest import ROOT
from delta_feedback_experiment_b200 import _lib, build


@pytest.fixture(scope="module")
def lib():
    build.build()
    return _lib.load()


def declared_functions():
    text = open(os.path.join(ROOT, "include", "pkda_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(pkda_[a-z0-9_]+)\s*\(", text)))


def test_header_symbols_exported(lib):
    names = declared_functions()
    assert set(names) == set(_lib.EXPORTS)
    for name in names:
        assert hasattr(lib, name), name


def test_struct_layouts(lib):
    assert lib.pkda_sizeof_problem() == C.sizeof(_lib.Problem)
    assert lib.pkda_sizeof_recurrent_args() == C.sizeof(_lib.RecurrentArgs)
    assert lib.pkda_sizeof_chunk_fwd_args() == C.sizeof(_lib.ChunkFwdArgs)
    assert lib.pkda_sizeof_chunk_bwd_args() == C.sizeof(_lib.ChunkBwdArgs)
    assert lib.pkda_abi_version() == _lib.ABI_VERSION


def test_status_codes_without_launch(lib):
    args = _lib.RecurrentArgs()
    args.p.n_seqs, args.p.seq_len, args.p.total_tokens = 2, 4, 8
    args.p.heads, args.p.head_dim = 2, 128
    assert lib.pkda_recurrent_fwd(C.byref(args), None) == 1  # PKDA_ERR_NULL
    args.p.total_tokens = 7
    assert lib.pkda_recurrent_fwd(C.byref(args), None) == 2  # PKDA_ERR_SHAPE
    # empty problems are accepted and launch nothing
    args.p.n_seqs, args.p.seq_len, args.p.total_tokens = 0, 4, 0
    assert lib.pkda_recurrent_fwd(C.byref(args), None) == 0
    assert lib.pkda_last_launch_count() == 0
    cf = _lib.ChunkFwdArgs()
    cf.p.n_seqs, cf.p.seq_len, cf.p.total_tokens, cf.p.heads, cf.p.head_dim = 1, 64, 64, 1, 64
    for f in ("q", "k", "v", "g", "g_atk", "beta_atk", "beta", "A_log", "dt_bias", "log_atk_scale"):
        setattr(cf.p, f, 256)
    assert lib.pkda_chunk_fwd(C.byref(cf), None) == 2  # head_dim 64 unsupported by the chunked path
    assert b"geometry" in lib.pkda_status_string(2)
    assert _lib.load().pkda_chunk_fwd_workspace_bytes(C.byref(cf.p)) > 0


def test_operators_refuse_cpu_tensors():
    import torch
    from delta_feedback_experiment_b200 import fused_recurrent_precond_kda
    t = torch.zeros(1, 1, 1, 8)
    s = torch.zeros(1, 1, 1)
    with pytest.raises(RuntimeError, match="no CPU path"):
        fused_recurrent_precond_kda(t, t, t, t, s, s, s, torch.zeros(1), torch.zeros(8),
                                    log_atk_scale=torch.zeros(1))


def test_variant_switch_and_status_offsets(lib):
    """The testing switch accepts exactly the stages that have two implementations, and
    the status word sits inside the workspace the size query reports."""
    for name in (b"intra_fwd", b"scan_fwd", b"out_fwd", b"scan_bwd", b"intra_bwd"):
        assert lib.pkda_set_variant(name, 1) == 0
        assert lib.pkda_set_variant(name, 0) == 0
    assert lib.pkda_set_variant(b"atk_local", 1) == 2
    assert lib.pkda_set_variant(None, 1) == 1
    p = _lib.Problem()
    p.n_seqs, p.seq_len, p.total_tokens, p.heads, p.head_dim = 2, 130, 260, 3, 128
    for size, off in ((lib.pkda_chunk_fwd_workspace_bytes, lib.pkda_chunk_fwd_status_offset),
                      (lib.pkda_chunk_bwd_workspace_bytes, lib.pkda_chunk_bwd_status_offset)):
        total, where = size(C.byref(p)), off(C.byref(p))
        assert 0 < where and where + 4 <= total and where % 256 == 0


class _FakeTensor:
    """Stands in for a CUDA tensor where there is no GPU: only the attributes the
    device checks read."""

    def __init__(self, device):
        import torch
        self.is_cuda = device is not None
        self.device = torch.device("cuda", device) if device is not None else torch.device("cpu")


def test_arguments_on_different_devices_are_rejected_before_any_launch():
    from delta_feedback_experiment_b200 import ops
    ops._require_cuda(_FakeTensor(1), None, _FakeTensor(1))
    with pytest.raises(RuntimeError, match="different devices"):
        ops._require_cuda(_FakeTensor(0), _FakeTensor(1))
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops._require_cuda(_FakeTensor(0), _FakeTensor(None))
    calls = []
    guarded = ops._on_tensor_device(lambda first: calls.append(first))
    with pytest.raises(RuntimeError, match="no CPU path"):
        guarded(_FakeTensor(None))
    assert not calls


def test_intermediate_contract_check_names_the_offender():
    """`fla_ops._check_intermediates` compares what a forward returns with what the fake
    implementation promises (reference: fla_ops.py:100-128): count, shape, dtype, contiguity."""
    import pytest
    import torch
    from delta_feedback_experiment_b200 import fla_ops

    q = torch.empty(2, 130, 3, 128, dtype=torch.bfloat16)
    v = torch.empty(2, 130, 3, 128, dtype=torch.bfloat16)
    for lean in (True, False):
        good = [torch.empty(s, dtype=d) for s, d in fla_ops._intermediate_meta(q, v, lean)]
        fla_ops._check_intermediates(good, q, v, lean)                       # passes
        with pytest.raises(RuntimeError, match="intermediates where"):
            fla_ops._check_intermediates(good[:-1], q, v, lean)
        bad = list(good)
        bad[2] = bad[2].float()                                               # wrong dtype
        with pytest.raises(RuntimeError, match="k_precond"):
            fla_ops._check_intermediates(bad, q, v, lean)
        bad = list(good)
        bad[0] = good[0].transpose(1, 2).contiguous().transpose(1, 2)         # right shape, not contiguous
        with pytest.raises(RuntimeError, match="Aqk"):
            fla_ops._check_intermediates(bad, q, v, lean)
    assert len(fla_ops._intermediate_meta(q, v, True)) == len(fla_ops.PKDA_INTERMEDIATES)
    assert fla_ops._intermediate_meta(q, v, False)[9][0] == (2, 3, 3, 128, 128)   # h: three chunks of 64


def test_intermediate_contract_check_agrees_with_the_fake_implementation():
    """The check on the operator's path and the list promised to a compiler are written in two
    languages: they must agree over batches, ragged lengths, head widths and both dtypes."""
    import torch
    from delta_feedback_experiment_b200 import _lib, fla_ops

    for B, T, H, D in ((1, 1, 1, 128), (3, 64, 2, 128), (2, 65, 5, 128), (1, 200, 4, 8), (2, 129, 1, 64)):
        for dtype in (torch.bfloat16, torch.float32):
            q = torch.empty(B, T, H, D, dtype=dtype, device="meta")
            for lean in (True, False):
                promised = [torch.empty(s, dtype=d, device="meta") for s, d in fla_ops._intermediate_meta(q, q, lean)]
                _lib.native().check_intermediates(promised, q, q, lean)
                with pytest.raises(RuntimeError, match="missing"):
                    _lib.native().check_intermediates([*promised[:-1], None], q, q, lean)


def test_exact_pair_refuses_misaligned_buffers_without_launch(lib):
    """Their kernels move states four floats at a time: a misaligned buffer is an error code, not a fault."""
    def problem(args):
        p = args.p
        p.n_seqs, p.seq_len, p.total_tokens, p.heads, p.head_dim, p.dtype = 1, 8, 8, 1, 32, _lib.PKDA_F32
        for f in ("q", "k", "v", "g", "g_atk", "beta_atk", "beta", "A_log", "dt_bias", "log_atk_scale"):
            setattr(p, f, 256)
        return p

    fwd = _lib.RecurrentArgs()
    p = problem(fwd)
    fwd.o = 256
    need = lib.pkda_recurrent_saved_bytes(C.byref(p))
    assert lib.pkda_recurrent_fwd_saving(C.byref(fwd), 264, need, None) == 6
    bwd = _lib.RecurrentBwdArgs()
    p = problem(bwd)
    for f in ("d_o", "dq", "dk", "dv", "dg", "dg_atk", "dbeta_atk", "dbeta", "dA_log", "ddt_bias", "dlog_atk_scale"):
        setattr(bwd, f, 256)
    bwd.workspace, bwd.workspace_bytes = 256, lib.pkda_recurrent_bwd_workspace_bytes(C.byref(p))
    assert lib.pkda_recurrent_bwd_saved(C.byref(bwd), 264, need, None) == 6
    bwd.workspace = 260
    assert lib.pkda_recurrent_bwd(C.byref(bwd), None) == 6
    assert lib.pkda_last_launch_count() == 0


def _chunk_args(args, size_query, units, pointers):
    """Arguments of a dense call of `units` rows of 64 tokens, one head, every buffer on a 256-byte boundary."""
    p = args.p
    p.n_seqs, p.seq_len, p.total_tokens, p.heads, p.head_dim = units, 64, 64 * units, 1, 128
    for f in ("q", "k", "v", "g", "g_atk", "beta_atk", "beta", "A_log", "dt_bias", "log_atk_scale"):
        setattr(p, f, 256)
    for f in pointers:
        setattr(args, f, 256)
    args.workspace, args.workspace_bytes = 256, size_query(C.byref(p))
    return args


FWD_POINTERS = ("o", "final_state", "final_A_state", "Aqk", "Akk", "k_precond", "ac_atk", "a_atk", "sa_atk", "w", "kg",
                "v_new", "h", "qg")
BWD_POINTERS = ("d_o", "d_final_state", "Aqk", "Akk", "k_precond", "ac_atk", "a_atk", "sa_atk", "w", "kg", "v_new", "h", "qg",
                "dq", "dk", "dv", "dg", "dg_atk", "dbeta_atk", "dbeta", "dA_log", "ddt_bias", "dlog_atk_scale",
                "d_initial_state", "d_initial_A_state")


def test_chunked_pair_refuses_misaligned_buffers_without_launch(lib):
    """Every buffer that a kernel of the chunked path moves several values at a time, or by TMA.  Few units take
    the column scans, which touch the states by scalars, and many the tensor-memory scans, which do not.
    (Only calls that are refused: these addresses must never reach a kernel.)"""
    always = [("o", 4), ("Aqk", 8), ("Akk", 8), ("k_precond", 4), ("ac_atk", 4), ("ac_atk", 8), ("w", 8), ("kg", 8),
              ("v_new", 4), ("h", 4), ("qg", 8), ("workspace", 8), ("p.dt_bias", 4)]
    many = [("final_state", 4), ("v_new", 8), ("h", 8)]
    for units, cases in ((2, always), (200, [c for c in always if c[0] != "o"] + many)):
        for name, off in cases:
            a = _chunk_args(_lib.ChunkFwdArgs(), lib.pkda_chunk_fwd_workspace_bytes, units, FWD_POINTERS)
            setattr(a.p if name[:2] == "p." else a, name.removeprefix("p."), 256 + off)
            assert lib.pkda_chunk_fwd(C.byref(a), None) == 6, (units, name, off)
    always = [(n, 8) for n in ("d_o", "Aqk", "Akk", "k_precond", "ac_atk", "a_atk", "w", "kg", "v_new", "h", "qg", "dv", "dg",
                               "workspace", "p.dt_bias")] + [("a_atk", 4), ("dk", 4), ("dq", 2)]
    for units, cases in ((2, always), (200, [*always, ("d_final_state", 4), ("d_initial_state", 8)])):
        for name, off in cases:
            a = _chunk_args(_lib.ChunkBwdArgs(), lib.pkda_chunk_bwd_workspace_bytes, units, BWD_POINTERS)
            a.recompute = 1
            setattr(a.p if name[:2] == "p." else a, name.removeprefix("p."), 256 + off)
            assert lib.pkda_chunk_bwd(C.byref(a), None) == 6, (units, name, off)
    assert lib.pkda_last_launch_count() == 0


@pytest.mark.parametrize("rows,T", [(2, 1), (200, 2), (2000, 40)])
def test_token_by_token_forward_refuses_a_misaligned_final_state(lib, rows, T):
    """The single step, the few-token kernel and the scan with four columns per lane write states by float4."""
    a = _lib.RecurrentArgs()
    p = a.p
    p.n_seqs, p.seq_len, p.total_tokens, p.heads, p.head_dim = rows, T, rows * T, 1, 128
    for f in ("q", "k", "v", "g", "g_atk", "beta_atk", "beta", "A_log", "dt_bias", "log_atk_scale", "initial_state"):
        setattr(p, f, 256)
    a.o, a.final_state = 256, 260
    assert lib.pkda_recurrent_fwd(C.byref(a), None) == 6
    assert lib.pkda_last_launch_count() == 0
