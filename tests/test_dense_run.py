"""What the native launches of layer runs ask of their description, without a GPU."""

import ctypes

import pytest


def test_the_records_are_as_long_as_their_description(monkeypatch):
    """A field on one side only would shift device pointers; the launch refuses instead."""
    from tokamak_b200.csrc import ops
    from tokamak_b200.csrc.lib import library
    assert ctypes.sizeof(ops.DenseStep) == library().tk_dense_step_bytes()
    fields = library().tk_dense_layer_bytes() // ctypes.sizeof(ctypes.c_void_p)

    class Longer(ops.DenseStep):
        _fields_ = [("more", ctypes.c_int)]

    for step, n in ((Longer(), fields), (ops.DenseStep(), fields + 1), (ops.DenseStep(), fields - 1)):
        with monkeypatch.context() as m:
            m.setattr(ops, "DenseStep", type(step))
            with pytest.raises(ops.KernelError, match="differ in size"):
                ops._want_dense_records(n)
            m.setattr(ops, "_DENSE_RECORDS_AGREE", False)
            with pytest.raises(ops.KernelError, match="differ in size"):
                ops.dense_layers([], [None] * n, step)
