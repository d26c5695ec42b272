"""The expression kernels compile: every operation over every pair of column types (no GPU needed)."""

import ctypes as C

import numpy as np
import pytest

from polars_b200 import _abi as A
from polars_b200._native import ColumnData, _arith_wire, _to_abi_columns, compile_predicate
from test_jit_cpu import _lib, nvrtc_available

pytestmark = pytest.mark.skipif(not nvrtc_available(), reason="NVRTC not installed")


@pytest.mark.parametrize("op", ["Add", "Sub", "Mul", "TrueDiv", "FloorDiv", "Mod"])
def test_expression_kernels_compile(op):
    names = [f"c{i}" for i in range(10)]
    types = ["int8", "uint8", "int16", "uint16", "int32", "uint32", "int64", "uint64", "float32", "float64"]
    cols = [ColumnData(np.ones(32, t), np.full(4, 255, np.uint8) if i % 2 else None) for i, t in enumerate(types)]
    abi, keep = _to_abi_columns(cols)
    fn = _lib().pmb_debug_jit_compile_expr
    fn.argtypes = [C.POINTER(A.Expr), C.POINTER(A.Column), C.c_int32, C.c_char_p, C.c_int64]
    buf = C.create_string_buffer(1 << 16)
    for i in range(10):
        other = {"kind": "LiteralF64", "value": 1.5} if i == 3 else {"kind": "LiteralI64", "value": -7} if i == 4 else \
            {"kind": "Column", "name": names[(i * 3 + 2) % 10]}
        e = _arith_wire({"kind": "Arith", "op": op, "lhs": {"kind": "Column", "name": names[i]}, "rhs": {
            "kind": "Arith", "op": op, "lhs": other, "rhs": {"kind": "Column", "name": names[(i + 5) % 10]}}})
        expr, ek = compile_predicate(e, {n: j for j, n in enumerate(names)})
        rc = fn(C.byref(expr), abi, len(cols), buf, 1 << 16)
        assert rc == 0, buf.value.decode()
    del keep
