"""Calls inside a caller's own CUDA-graph capture, after a call that has made
the engine's buffers.  Each case runs in a process of its own: a capture that
fails leaves the capturing library in whatever state it has for it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HEAD = """
import ctypes, glob, os
import torch
import highuvlith_b200 as HB

def engine(n=256):
    return HB.SimulationEngine(HB.SourceConfig.euv(0.5), HB.OpticsConfig.euv_nxe_033(), grid=HB.GridConfig(n, 1.0),
                               max_kernels=8)

def copies(graph):  # memcpy nodes
    rt = ctypes.CDLL(None)
    if not hasattr(rt, "cudaGraphGetNodes"):
        import nvidia.cuda_runtime as r
        rt = ctypes.CDLL(glob.glob(os.path.join(list(r.__path__)[0], "lib", "libcudart.so*"))[0])
    count, kind = ctypes.c_size_t(), ctypes.c_int()
    handle = ctypes.c_void_p(graph.raw_cuda_graph())
    assert rt.cudaGraphGetNodes(handle, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert rt.cudaGraphGetNodes(handle, nodes, ctypes.byref(count)) == 0
    found = 0
    for n in nodes:
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(n), ctypes.byref(kind)) == 0
        found += kind.value == 1
    return found
"""


def _run(body):
    r = subprocess.run([sys.executable, "-c", HEAD + body], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return r.stdout.split()


def test_rectangle_clips_leave_no_copy_of_host_memory_in_the_graph():
    """The engine's staging vector moves with later calls: a copy node would
    read it wherever it was."""
    assert _run("""
eng = engine()
clips = [[(0.0, 0.0, 60.0, 40.0), (50.0, 10.0, 20.0, 90.0)], [(-30.0, 0.0, 30.0, 30.0)]]
out = torch.empty((2, 256, 256), device="cuda")
ref = eng.compute_batch_rects(clips).clone()
eng.compute_batch_rects(clips, out=out)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph(keep_graph=True)
with torch.cuda.graph(g):
    eng.compute_batch_rects(clips, out=out)
print(copies(g))
g.instantiate()
out.zero_()
g.replay()
torch.cuda.synchronize()
print(torch.equal(out, ref))
""") == ["0", "True"]


@pytest.mark.parametrize("n", [256, 512, 1024])
def test_real_masks_after_complex_maps_only(n):
    """Complex maps have made every buffer that the real masks need but the
    folded kernels, which a capture cannot make: it takes the set as it is."""
    assert _run(f"""
eng, n = engine({n}), {n}
x = (torch.rand(1, n // 8, n // 8, device="cuda") > 0.5).to(torch.uint8).repeat_interleave(8, 1).repeat_interleave(8, 2)
c = x.to(torch.complex64)
out = torch.empty((1, n, n), device="cuda")
eng.compute_batch(c, out=out)
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
with torch.cuda.graph(g):
    eng.compute_batch(x, out=out)
out.zero_()
g.replay()
torch.cuda.synchronize()
ref = eng.compute_batch(x)  # folded
print(float((out - ref).abs().max() / ref.max()) < 5e-6)  # two FP32 evaluations, each within 2e-6
""") == ["True"]
