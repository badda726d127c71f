"""What crosses to the kernels' C functions as an int, and what they may read early."""
import ctypes
import inspect

import pytest
import torch

from ember_b200 import ops


@pytest.mark.parametrize("value", [2.0, 2.5, "3", None, torch.tensor(1.5)])
def test_what_is_no_whole_number_is_refused(value):
    for convert in (ctypes.c_int, ops.c_int):
        with pytest.raises(TypeError):
            convert(value)


@pytest.mark.parametrize("value", [0, -3, True, 2 ** 31 - 1, torch.tensor(7)])
def test_whole_numbers_arrive(value):
    assert ctypes.c_int(ops.c_int(value)).value == ctypes.c_int(value).value


@pytest.mark.parametrize("op,name", [("attention_tc", "keys_settled"), ("gemm_simt", "weights_settled")])
def test_early_reads_are_asked_for(op, name):
    """A kernel reads ahead of the kernel before it only where its caller says that it may."""
    assert inspect.signature(getattr(ops, op)).parameters[name].default is False


@pytest.mark.parametrize("tokens,rows,fused", [(1, 14336, True), (24, 14336, True), (25, 7168, True), (25, 7296, False), (64, 7168, True), (65, 7168, False),
                                               (65, 4096, True), (128, 4096, True), (128, 4224, False), (129, 4096, False)])
def test_where_the_product_finishes_the_heads(tokens, rows, fused):
    assert ops.qkv_fuse_few(tokens, rows) is fused


def test_where_gate_norm_and_norm_are_one_kernel():
    whole, odd = torch.zeros(9)[:8], torch.zeros(9)[1:]
    assert whole.data_ptr() % 16 == 0
    assert ops.gated_norm_add_norm_usable(8192, None, whole, None, whole)
    assert not ops.gated_norm_add_norm_usable(2048, whole, odd)
    assert not any(ops.gated_norm_add_norm_usable(w, whole) for w in (0, 2, 2050, 8196))


class _Recorder:
    """Stands for a compiled library: keeps the arguments of the last call of each function."""

    def __init__(self):
        self.calls = {}

    def __getattr__(self, name):
        def call(*args):
            self.calls[name] = [getattr(a, "value", a) for a in args]
            return 0
        return call


def test_attention_beside_portions_only_directly_behind_them(monkeypatch):
    """The decode kernel is handed the ticket of the portions' kernel (its word and number) only if nothing was launched
    between the two, on the same stream; otherwise it gets none and waits like any other kernel."""
    lib = _Recorder()
    monkeypatch.setattr(ops, "_lib", lambda name: lib)
    monkeypatch.setattr(ops, "_check", lambda t, name, dtype=None: None)
    pool, q, ints = torch.zeros(2, 1, 16, 128, dtype=torch.bfloat16), torch.zeros(4, 128, dtype=torch.bfloat16), torch.zeros(4, 4, dtype=torch.int32)

    def portions(stream, late=True):
        ops.attention_fa(q, pool, pool, q, 1, 1, 128, ints, 1, ints, 16, 0, 0.1, stream=stream, release_late=late)
        return tuple(lib.calls["ember_attention_fa"][-3:-1])

    def decoded(stream, beside=True):
        ops.attention_tc(q, pool, pool, q, 1, 1, 1, 128, ints, 1, ints, 16, 0, 0.1, stream=stream, beside=beside)
        return tuple(lib.calls["ember_attention_tc"][-3:-1])

    none = (None, 0)
    first = portions(7)
    assert first[0] and first[1] and decoded(7) == first
    assert decoded(7) == none                                     # (another launch lies between)
    second = portions(7)
    assert second[1] != first[1] and decoded(8) == none           # (another stream)
    portions(7)
    ops.embed(ints[0], torch.zeros(2, 8), torch.zeros(4, 8), stream=7)
    assert decoded(7) == none
    portions(7)
    assert decoded(7, beside=False) == none
    assert portions(7, late=False) == none and decoded(7) == none
