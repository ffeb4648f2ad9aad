"""Results of plane-cut batches that are alive at the same time, outlive their
handle or are released in either order keep their halves, whichever of them
holds the handle's readback buffer; device meshes that are neighbours in the
cut's buffers, alone or apart give the hulls of the same meshes on the host."""
import ctypes as C

import numpy as np
import pytest

from conftest import pkg

A, G, T = pkg("_abi"), pkg("meshgen"), pkg("tree")

pytestmark = pytest.mark.gpu


def cut(g, m, planes):
    pl = np.ascontiguousarray(planes, np.float64)
    idx = np.zeros(len(pl), np.int32)
    h = C.c_void_p()
    ma = A.MeshArray([m])
    assert T.load_library().cuacd_tree_plane_cuts(g.h, ma.arr, 1, idx.ctypes.data_as(C.POINTER(C.c_int32)),
                                                  pl.ctypes.data_as(C.POINTER(C.c_double)), len(pl), 0, C.byref(h)) == 0
    return h


def halves(h, n):
    """(verts, tris) of every half through the call for one of them, with their device copies' addresses"""
    L = T.load_library()
    L.cuacd_cuts_half_device.argtypes = [C.c_void_p, C.c_int, C.c_int, C.POINTER(C.POINTER(C.c_float)),
                                         C.POINTER(C.POINTER(C.c_uint32))]
    out, dev = [], []
    for k in range(2 * n):
        v, t, nv, nt = C.POINTER(C.c_float)(), C.POINTER(C.c_uint32)(), C.c_uint32(), C.c_uint32()
        dv, dt = C.POINTER(C.c_float)(), C.POINTER(C.c_uint32)()
        if L.cuacd_cuts_half(h, k // 2, k % 2, C.byref(v), C.byref(nv), C.byref(t), C.byref(nt)) != 0:
            out.append(None)
            dev.append(None)
            continue
        assert L.cuacd_cuts_half_device(h, k // 2, k % 2, C.byref(dv), C.byref(dt)) == 0
        out.append((np.ctypeslib.as_array(v, (nv.value * 3,)).copy(), np.ctypeslib.as_array(t, (nt.value * 3,)).copy()))
        dev.append((dv, dt, nv.value, nt.value))
    return out, dev


def same(a, b):
    return all((x is None) == (y is None) and (x is None or (np.array_equal(x[0], y[0]) and np.array_equal(x[1], y[1])))
               for x, y in zip(a, b))


def sphere(level, seed):
    m = G.noisy_icosphere(level, seed=seed)
    return T.Mesh(m.verts - (m.verts.min(0) + m.verts.max(0)) / 2, m.tris)


PLANES = [[1.0, 0, 0, 0.05], [0, 1.0, 0, 9.0], [0, 0, 1.0, -0.1], [0.6, 0.8, 0, 0]]  # the second misses the mesh


@pytest.mark.parametrize("first_out,close", [(True, False), (False, False), (True, True), (False, True)])
def test_results_alive_together(first_out, close):
    L = T.load_library()
    g = T.GpuTree(width=3, depth=1, hullMaxVerts=4096)
    ms = [sphere(k, k) for k in (2, 4, 3)]
    want = []
    for m in ms:
        r = g.plane_cuts([m], PLANES, [0] * len(PLANES))
        assert [x[0] for x in r] == [0, 1, 0, 0]
        want.append([None if x[0] else (h.verts.ravel(), h.tris.ravel()) for x in r for h in (x[1:] if x[0] == 0 else (0, 0))])
    hs = [cut(g, m, PLANES) for m in ms[:2]]
    assert all(same(halves(h, 4)[0], w) for h, w in zip(hs, want))
    L.cuacd_cuts_free(hs.pop(0 if first_out else 1))
    kept = 1 if first_out else 0
    hs.append(cut(g, ms[2], PLANES))
    if close:
        g.destroy()
    assert same(halves(hs[0], 4)[0], want[kept]) and same(halves(hs[1], 4)[0], want[2])
    for h in hs:
        L.cuacd_cuts_free(h)


@pytest.mark.parametrize("order", [[0, 1, 4, 5, 6, 7], [7, 6, 5, 4, 1, 0], [0, 1, 5, 4, 6], [4], ["host", 0, 1, "host", 4, 5]])
def test_neighbours_on_the_device(order):
    L = T.load_library()
    g = T.GpuTree(width=3, depth=1, hullMaxVerts=4096)
    h = cut(g, sphere(3, 3), PLANES)
    host, dev = halves(h, 4)
    other = G.staircase(3)
    ms = [other if k == "host" else T.Mesh(*(x.reshape(-1, 3) for x in host[k])) for k in order]
    ref = A.MeshArray(ms)
    for i, k in enumerate(order):
        if k != "host":
            ref.arr[i].verts, ref.arr[i].tris, ref.arr[i].nv, ref.arr[i].nt = dev[k]
    n, stride = len(order), 6 * max(m.nv for m in ms)
    tris, vol = np.zeros(n * stride, np.uint32), np.zeros(n, np.float32)
    nt, st = np.zeros(n, np.uint32), np.zeros(n, np.int32)
    assert L.cuacd_tree_hull_meshes(g.h, ref.arr, n, 0, A.uptr(tris), stride, A.fptr(vol), A.uptr(nt),
                                    st.ctypes.data_as(C.POINTER(C.c_int32))) == 0
    for k in range(n):  # the meshes as they were uploaded
        v, t, _ = g.part_geometry(k)
        assert np.array_equal(v, ms[k].verts) and np.array_equal(t, ms[k].tris)
    L.cuacd_cuts_free(h)
    want, _ = g.hull_meshes(ms)
    for k in range(n):
        assert st[k] == 0 and vol[k] == want[k]["volume"]
        assert np.array_equal(tris[k * stride: k * stride + 3 * nt[k]].reshape(-1, 3), want[k]["tris"])
