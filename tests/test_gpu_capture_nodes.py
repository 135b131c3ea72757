"""A captured assembly call is kernels only: the graph can stand in another graph and have several executable copies, and
its replays have the bits of the call.  Its workspace goes when the graph goes."""
import ctypes as C

import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, perturbed_vertices

CFGS = {
    "nonlinear_q1": dict(dim=3, order=1, n=(20, 19, 18), kind="diffusion_1pu2"),
    "general_q1": dict(dim=3, order=1, n=(9, 8, 7), kind="diffusion_1pu2",
                       vertex_coords=perturbed_vertices(3, (9, 8, 7), (0, 0, 0), (1, 1, 1), 0.2, 3)),
    "quad_q2": dict(dim=2, order=2, n=(30, 20), kind="diffusion_1pu2"),
    "nonlinear_q2": dict(dim=3, order=2, n=(9, 8, 7), kind="diffusion_1pu2"),
    "nonlinear_q2_slabs": dict(dim=3, order=2, n=(41, 40, 39), kind="diffusion_1pu2"),
}
MEM_ALLOC, MEM_FREE = 10, 11  # cudaGraphNodeType


@pytest.fixture(scope="module")
def rt(cuda):
    return C.CDLL("libcudart.so." + torch.version.cuda.split(".")[0])


def _node_types(rt, graph):
    n = C.c_size_t(0)
    assert rt.cudaGraphGetNodes(graph, None, C.byref(n)) == 0
    nodes = (C.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, C.byref(n)) == 0
    out = []
    for k in nodes:
        t = C.c_int(-1)
        assert rt.cudaGraphNodeGetType(C.c_void_p(k), C.byref(t)) == 0
        out.append(t.value)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CFGS))
@pytest.mark.parametrize("fp32", [False, True])
def test_captured_assembly_is_kernels_only(rt, name, fp32):
    from mrhyde_gb300 import AssemblyManager

    G = gpu_problem(CFGS[name])
    A = AssemblyManager(G)
    u = torch.tensor(np.random.default_rng(9).uniform(0.0, 0.5, G.info.n_dofs), device="cuda")
    r, J = G.new_vector(), G.new_matrix_values(fp32=fp32)

    def run():  # two calls share the stream's workspace
        A.assembleJacRes(u, r, J, fp32_jacobian=fp32, overwrite=True)
        A.assembleJacRes(u, r, J, fp32_jacobian=fp32)

    run()
    want = r.clone(), J.clone()
    stream = torch.cuda.Stream()
    graph, parent = C.c_void_p(), C.c_void_p()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        s = C.c_void_p(stream.cuda_stream)
        assert rt.cudaStreamBeginCapture(s, 0) == 0
        run()
        assert rt.cudaStreamEndCapture(s, C.byref(graph)) == 0
    assert not {MEM_ALLOC, MEM_FREE} & set(_node_types(rt, graph))
    # as a part of another graph, of which there are two executable copies
    node, execs = C.c_void_p(), [C.c_void_p(), C.c_void_p()]
    assert rt.cudaGraphCreate(C.byref(parent), 0) == 0
    assert rt.cudaGraphAddChildGraphNode(C.byref(node), parent, None, C.c_size_t(0), graph) == 0
    for e in execs:
        assert rt.cudaGraphInstantiate(C.byref(e), parent, C.c_ulonglong(0)) == 0
    assert rt.cudaGraphDestroy(graph) == 0 and rt.cudaGraphDestroy(parent) == 0
    for e in execs:
        r.fill_(7.0)
        J.fill_(7.0)
        torch.cuda.synchronize()
        assert rt.cudaGraphLaunch(e, s) == 0
        A.assembleRes(u, torch.empty_like(r), overwrite=True)  # beside it, with a workspace of its own
        torch.cuda.synchronize()
        assert torch.equal(r, want[0]) and torch.equal(J, want[1])
    for e in execs:
        assert rt.cudaGraphExecDestroy(e) == 0
    G.close()


@pytest.mark.gpu
def test_workspaces_of_captures_go_with_their_graphs(cuda):
    from mrhyde_gb300 import AssemblyManager

    G = gpu_problem(dict(dim=3, order=1, n=(60, 60, 60), kind="diffusion_1pu2"))  # 107 MB in FP64
    A = AssemblyManager(G)
    u, r, J = G.new_vector(), G.new_vector(), G.new_matrix_values()
    free = []
    for _ in range(12):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            A.assembleJacRes(u, r, J, overwrite=True)
        g.replay()
        torch.cuda.synchronize()
        free.append(torch.cuda.mem_get_info()[0])  # the next capture begins where this graph's workspace is given back
        del g
    assert free[2] - free[-1] <= 250e6  # the nine between would be 960 MB
    G.close()
