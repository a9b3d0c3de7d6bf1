"""Calls without a stream run on the stream that is current in torch at the call:
the default one, one of a context, one inside another, and again the outer one."""
import pytest

from morganapublic_gb300 import meshgen

pytestmark = pytest.mark.gpu


def test_current_stream_is_followed():
    import torch

    import morganapublic_gb300 as mg
    m = meshgen.kuhn_cube(4)
    b = mg.MatrixBuilder(mg.Mesh(m.xyz, m.conn))
    want = b.assemble("stiff_const")
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    assert mg._stream_ptr(None) == torch.cuda.current_stream().cuda_stream
    for s in streams:
        with torch.cuda.stream(s):
            assert mg._stream_ptr(None) == s.cuda_stream
            with torch.cuda.stream(streams[0]):
                assert mg._stream_ptr(None) == streams[0].cuda_stream
            assert mg._stream_ptr(None) == s.cuda_stream
            got = b.assemble("stiff_const")
            s.synchronize()  # the call's work is on s: nothing is left after this
            assert bool((got == want).all())
    assert mg._stream_ptr(None) == torch.cuda.current_stream().cuda_stream
    assert mg._stream_ptr(streams[1]) == streams[1].cuda_stream and mg._stream_ptr(7) == 7
