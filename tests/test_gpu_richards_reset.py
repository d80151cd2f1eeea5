"""A reset of a Richards line empties the exchange slots of its one-launch step: a step that gave up waiting
leaves values in them, which the next run would take for its own. Seen in the work that the reset enqueues
(captured into a graph): a clear of 32 doubles per chunk to all ones."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_richards_step import _case

pytestmark = pytest.mark.gpu


class _Memset(C.Structure):
    _fields_ = [("dst", C.c_void_p), ("pitch", C.c_size_t), ("value", C.c_uint), ("elementSize", C.c_uint),
                ("width", C.c_size_t), ("height", C.c_size_t)]


def test_reset_empties_the_slots():
    torch = pytest.importorskip("torch")
    import fpde_hpc_gb300 as fp
    rt = C.CDLL("libcudart.so")
    ok = lambda rc: rc == 0 or pytest.fail(f"CUDA call failed: {rc}")
    N, steps = 1000, 10
    c = _case(N, steps, False)
    with fp.Context(0) as ctx:
        line = fp.Line(ctx, N, c["alpha"], c["tau"], c["Da"], None, None, None, c["u0"], steps, right=(0, c["u0"][-1]),
                       richards=dict(k_form=1, k_sat=2e-6, Z=c["Z"], dL=c["dL"], evaporation=c["E"]))
        u0 = torch.from_numpy(c["u0"]).cuda()
        torch.cuda.synchronize()
        st, graph, n = C.c_void_p(), C.c_void_p(), C.c_size_t(0)
        ok(rt.cudaStreamCreateWithFlags(C.byref(st), 1))
        ctx.set_stream(st.value)
        ok(rt.cudaStreamBeginCapture(st, 1))
        line.reset(u0)
        ok(rt.cudaStreamEndCapture(st, C.byref(graph)))
        ctx.set_stream(None)
        ok(rt.cudaGraphGetNodes(graph, None, C.byref(n)))
        nodes = (C.c_void_p * n.value)()
        ok(rt.cudaGraphGetNodes(graph, nodes, C.byref(n)))
        clears = []
        for node in nodes:
            kind, par = C.c_int(-1), _Memset()
            ok(rt.cudaGraphNodeGetType(C.c_void_p(node), C.byref(kind)))
            if kind.value == 2:                            # cudaGraphNodeTypeMemset
                ok(rt.cudaGraphMemsetNodeGetParams(C.c_void_p(node), C.byref(par)))
                clears.append((par.value & 0xFF, par.elementSize * par.width * max(par.height, 1)))
        rt.cudaGraphDestroy(graph)
        chunks = -(-(N - 1) // 32)
        assert (0xFF, 32 * chunks * 8) in clears, clears
        line.reset(c["u0"])                                # and the line still runs
        line.run(steps)
        assert np.isfinite(line.state()).all()
        line.close()
        rt.cudaStreamDestroy(st)
