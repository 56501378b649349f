"""What the library asks of the CUDA runtime, seen by a stand-in in front of it."""
import pytest

import cudart_shim

pytestmark = pytest.mark.gpu


def test_an_explicit_launch_shape_is_the_one_that_runs(tmp_path):
    # a mesh whose grid tiles fit the GPU all at once: by default one CTA per
    # tile, but persistent 0 and 1 launch their own kernels, and what is read
    # back sets the same again
    cudart_shim.run(tmp_path, r"""
ctx = pb.DeviceContext(pb.Mesh(RVE(nx=40, ny=30, strain=0.01)))
asm = pb.Assembler(ctx)
def one(tile, persistent):
    _lib.check(_lib.lib.pg_ctx_set_tuning(ctx.handle, tile, persistent, 4))
    return kernels(asm.assemble_linear)
tile, persistent, warps = C.c_int32(), C.c_int32(), C.c_int32()
_lib.check(_lib.lib.pg_ctx_tuning(ctx.handle, C.byref(tile), C.byref(persistent), C.byref(warps)))
default = kernels(asm.assemble_linear)
assert one(tile.value, persistent.value) == default
assert (tile.value, persistent.value) == (128, 0)
for t in (128, 256):
    assert one(t, 0) != one(t, 1), t
ctx.close()
""")
