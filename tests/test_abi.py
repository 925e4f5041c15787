"""The C-ABI library loads and exports exactly what `include/b200moe.h` declares."""

import ctypes
import re
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def declared_symbols():
    header = (ROOT / "include" / "b200moe.h").read_text()
    return sorted(set(re.findall(r"\b(b200moe_\w+)\s*\(", header)))


def test_header_declares_entry_points():
    names = declared_symbols()
    assert "b200moe_grouped_gemm_fp8" in names and "b200moe_route_topk" in names
    assert len(names) >= 12


def test_library_exports_every_declared_symbol():
    from mlops_b200 import _lib

    handle = ctypes.CDLL(str(_lib.LIBRARY_PATH))
    for name in declared_symbols():
        assert hasattr(handle, name), f"{name} is declared in the header but not exported"


def test_binding_covers_every_declared_symbol():
    from mlops_b200 import _lib

    assert sorted(_lib.SIGNATURES) == declared_symbols()


def test_argument_structs_are_laid_out_like_the_headers():
    """Field names, order and types of the argument structs agree with the C declarations."""
    from mlops_b200 import _lib

    text = re.sub(r"/\*.*?\*/", "", (ROOT / "include" / "b200moe.h").read_text(), flags=re.S)
    for name, struct in (("b200moe_forward_args", _lib.ForwardArgs), ("b200moe_backward_args", _lib.BackwardArgs)):
        body = re.search(r"typedef struct %s \{(.*?)\}" % name, text, flags=re.S).group(1)
        declared = []
        for line in body.split(";"):
            if not line.strip():
                continue
            if "*" in line:
                declared.append((line.split("*")[1].strip(), ctypes.c_void_p))
            else:
                kind = next(k for k in ("long long", "int", "float") if line.strip().startswith(k))
                ctype = {"long long": ctypes.c_longlong, "int": ctypes.c_int, "float": ctypes.c_float}[kind]
                declared += [(n.strip(), ctype) for n in line.strip()[len(kind):].split(",")]
        assert declared == list(struct._fields_)


def test_argument_validation_needs_no_gpu():
    """Entry points reject null pointers and bad sizes before touching the device."""
    from mlops_b200._lib import lib

    assert lib.b200moe_route_topk(None, 0, 1, 8, 2, 1, None, 1, 1, 1.0, None, None, None) == -1
    assert lib.b200moe_sort_assignments_workspace_bytes(4096 * 3 + 1, 8) == 4 * 8 * 4
    assert lib.b200moe_sort_assignments_workspace_bytes(-1, 8) == -1
    assert lib.b200moe_grouped_gemm_fp8(None, 0, None, 0, 0, None, None, None, 0, None, 0, None, 1, 1, 0, 8, 16, 0,
                                        128,
                                        None, None) == -1
    assert lib.b200moe_forward_fp8(None, None) == -1 and lib.b200moe_backward_fp8(None, None) == -1
    assert lib.b200moe_forward_workspace_bytes(4, 100, 128, 8, 2) == -1
    assert lib.b200moe_combine(None, 0, 0, None, None, None, 0, None, 0, 0, 8, 1, None) == -1


def test_the_layer_calls_refuse_every_missing_pointer_before_any_launch():
    """Each required pointer of the two layer calls cleared in turn, a mode out of range, a misaligned
    pointer: an error before the first launch, so the (invented) addresses are never used. Optional
    pointers are those the header lets a caller leave out."""
    from mlops_b200._lib import BackwardArgs, ForwardArgs, lib

    sizes = dict(tokens=4, width=256, inner=128, experts=8, top_k=2)
    for struct, call, optional in (
            (ForwardArgs, lib.b200moe_forward_fp8, {"bias"}),
            (BackwardArgs, lib.b200moe_backward_fp8,
             {"grad_aux", "grad_probability_sum", "grad_w13", "grad_w2"})):
        pointers = [name for name, kind in struct._fields_ if kind is ctypes.c_void_p]

        def filled(**changes):
            fields = {**sizes, "mode": 1, **{name: 4096 for name in pointers}, **changes}
            return ctypes.byref(struct(**fields))

        for name in pointers:
            if name not in optional:
                assert call(filled(**{name: None}), None) == -1, name
        assert call(filled(mode=3), None) == -1 and call(filled(mode=-1), None) == -1
        assert call(filled(tokens=0), None) == -1 and call(filled(inner=100), None) == -1
        for name in ("x", "h13", "workspace"):
            assert call(filled(**{name: 4096 + 8}), None) == -2, name


def test_ops_refuse_cpu_tensors():
    import pytest
    import torch

    from mlops_b200 import ops
    from mlops_b200._lib import NativeError

    with pytest.raises(NativeError):
        ops.route_topk(torch.zeros(4, 8), 2, "softmax_then_topk")
    with pytest.raises(NativeError):
        ops.quantize_rows(torch.zeros(4, 128, dtype=torch.bfloat16))


def test_device_probes_compile_for_sm_100a():
    """The stand-alone probes beside the kernels build with nvcc (nothing runs without a GPU)."""
    from mlops_b200 import probes

    names = sorted(p.stem for p in probes.PROBES.glob("*.cu"))
    assert "handshake" in names
    for name in names:
        assert probes.build(name).exists()
