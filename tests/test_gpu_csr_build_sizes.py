"""gbx_csr_build and gbx_degree_reorder against a stable numpy sort, at the sizes where the sort changes:
around one tile of its passes (6,144 elements) and of its removal of repeats (4,096), several tiles, id widths
with a different number of 8-bit digits, digits that are the same in every edge, ids with mask bits, input
arrays that are also the outputs, and arrays that start off a 16-byte boundary. Every result is exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ID = np.uint32(0x3FFFFFFF)


def reference(src, dst, w, V, symmetric, dedup, by_dst):
    if symmetric:
        src, dst = np.concatenate([src, dst]), np.concatenate([dst, src])
        w = None if w is None else np.concatenate([w, w])
    order = np.lexsort((dst, src)) if by_dst else np.argsort(src, kind="stable")
    s, d = src[order], dst[order]
    ww = np.ones(len(s), np.float32) if w is None else w[order]
    if dedup:
        keep = s != d
        keep[1:] &= (s[1:] != s[:-1]) | (d[1:] != d[:-1])
        s, d, ww = s[keep], d[keep], ww[keep].astype(np.uint32).astype(np.float32)
    deg, idx = np.zeros(V, np.uint32), np.zeros(V, np.uint32)
    v = s & ID
    first = np.flatnonzero(np.r_[True, v[1:] != v[:-1]]) if len(v) else np.zeros(0, np.int64)
    idx[v[first]] = first
    deg[v[first]] = np.diff(np.r_[first, len(v)])
    return deg, idx, s, d, ww


def build(lib_call, src, dst, w, V, symmetric, dedup, sort, *, device=None, offset=0, in_place=False, want_w=True):
    """gbx_csr_build on host arrays, or on device tensors `offset` elements into their storage."""
    import torch

    E = len(src)
    cap = max(1, 2 * E if symmetric else E)
    n = C.c_uint32()
    if device is None:
        put = lambda a: a.copy()  # noqa: E731
        room = lambda k, dt: np.zeros(k, dt)  # noqa: E731
        ptr = lambda a: None if a is None else a.ctypes.data  # noqa: E731
        get = lambda a: a  # noqa: E731
    else:
        def put(a):
            t = torch.zeros(len(a) + offset, dtype=torch.int32 if a.dtype == np.uint32 else torch.float32, device=device)
            t[offset:] = torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a)
            return t[offset:]

        def room(k, dt):
            return torch.zeros(k + offset, dtype=torch.int32 if dt == np.uint32 else torch.float32, device=device)[offset:]

        ptr = lambda a: None if a is None else a.data_ptr()  # noqa: E731
        get = lambda a: a.cpu().numpy().view(np.uint32) if a.dtype == torch.int32 else a.cpu().numpy()  # noqa: E731
    s, d = put(src), put(dst)
    ww = None if w is None else put(w)
    deg, idx = room(V, np.uint32), room(V, np.uint32)
    so, do = (s, d) if in_place else (room(cap, np.uint32), room(cap, np.uint32))
    wo = (ww if in_place and ww is not None else room(cap, np.float32)) if want_w else None
    lib_call("gbx_csr_build", E, ptr(s), ptr(d), ptr(ww), int(symmetric), int(dedup), sort, V, ptr(deg), ptr(idx), ptr(so), ptr(do),
             ptr(wo), C.byref(n), None)
    k = n.value
    return get(deg), get(idx), get(so)[:k], get(do)[:k], None if wo is None else get(wo)[:k]


def compare(got, want):
    for name, g, x in zip(("out_degree", "edges_idx", "src", "dst", "weight"), got, want):
        if g is not None:
            np.testing.assert_array_equal(g, x, err_msg=name)


def edges(E, V, seed, hub=0.3):
    rng = np.random.default_rng(seed)
    src = rng.integers(0, V, E, dtype=np.uint32)
    dst = rng.integers(0, V, E, dtype=np.uint32)
    src[rng.random(E) < hub] = V // 2  # a hub: long runs, repeats, self loops
    dst[rng.random(E) < hub / 3] = V // 2
    return src, dst, (rng.random(E) * 300).astype(np.float32)


@pytest.mark.parametrize("E", [0, 1, 2, 31, 4095, 4096, 4097, 6143, 6144, 6145, 12289, 300_001])
@pytest.mark.parametrize("V", [1, 2, 255, 257, 65_536, (1 << 22) + 3])
def test_sizes(gbx, cuda_device, E, V):
    from graphblox_gb300._lib import call

    src, dst, w = edges(E, V, E + V)
    for symmetric, dedup, sort, weights in ((0, 0, 0, True), (0, 0, 1, True), (0, 1, 1, True), (1, 1, 1, False), (1, 0, 0, True)):
        ww = w if weights else None
        want = reference(src, dst, ww, V, symmetric, dedup, sort == 1)
        compare(build(call, src, dst, ww, V, symmetric, dedup, sort, device=cuda_device), want)


@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("E,V", [(5000, 200), (50_000, 3000), (50_000, 200_000)])
def test_in_place_and_alignment(gbx, cuda_device, E, V, offset):
    from graphblox_gb300._lib import call

    src, dst, w = edges(E, V, 7)
    for dedup, sort in ((0, 0), (0, 1), (1, 1)):
        want = reference(src, dst, w, V, 0, dedup, sort == 1)
        compare(build(call, src, dst, w, V, 0, dedup, sort, device=cuda_device, offset=offset, in_place=True), want)
        compare(build(call, src, dst, w, V, 0, dedup, sort, in_place=True), want)
        compare(build(call, src, dst, None, V, 0, dedup, sort, want_w=False), want[:4])


@pytest.mark.parametrize("sort,dedup", [(0, 0), (1, 0), (1, 1)])
def test_mask_bits(gbx, cuda_device, sort, dedup):
    from graphblox_gb300._lib import call

    V = 5000
    src, dst, w = edges(40_000, V, 3)
    hint = (np.random.default_rng(4).integers(0, 4, V).astype(np.uint32)) << np.uint32(30)
    src, dst = src | hint[src], dst | hint[dst]
    want = reference(src, dst, w, V, 0, dedup, sort == 1)
    compare(build(call, src, dst, w, V, 0, dedup, sort, device=cuda_device), want)


def test_one_digit_everywhere(gbx, cuda_device):
    """Every source the same, destinations in one 256-id block: most passes have nothing to move."""
    from graphblox_gb300._lib import call

    V = 1 << 20
    rng = np.random.default_rng(1)
    dst = (rng.integers(0, 256, 20_000) + 0x51200).astype(np.uint32)
    src = np.full(20_000, 0x81234, np.uint32)
    w = np.arange(20_000, dtype=np.float32)
    for dedup, sort in ((0, 0), (0, 1), (1, 1)):
        compare(build(call, src, dst, w, V, 0, dedup, sort, device=cuda_device), reference(src, dst, w, V, 0, dedup, sort == 1))
    one = np.full(9000, 0x81234, np.uint32)
    compare(build(call, one, one, w[:9000], V, 0, 0, 1, device=cuda_device), reference(one, one, w[:9000], V, 0, 0, True))


def test_id_out_of_range(gbx, cuda_device):
    from graphblox_gb300._lib import call

    src, dst, w = edges(10_000, 1000, 5)
    dst[777] = 1000
    for dedup in (0, 1):
        with pytest.raises(gbx.GbxError):
            build(call, src, dst, w, 1000, 0, dedup, 1, device=cuda_device)
    el = gbx.EdgeList(1000, src.copy(), dst.copy())
    with pytest.raises(gbx.GbxError):
        gbx.degree_reorder(el, 1)
    np.testing.assert_array_equal(el.src, src)


@pytest.mark.parametrize("V,E", [(1, 0), (1, 3), (2, 1), (6143, 9), (6144, 50_000), (6145, 200_000), (300_000, 100_000)])
@pytest.mark.parametrize("lmode", [1, 2, 3, 4])
def test_reorder_sizes(gbx, cuda_device, V, E, lmode):
    src, dst, _ = edges(E, V, V + lmode)
    el = gbx.EdgeList(V, src.copy(), dst.copy())
    gbx.degree_reorder(el, lmode)
    deg = np.zeros(V, np.int64)
    if lmode != 2:
        deg += np.bincount(src, minlength=V)
    if lmode in (2, 3):
        deg += np.bincount(dst, minlength=V)
    if lmode == 4:
        avg = E // V
        t = [1 if avg <= 1 else avg // 2]
        t += [t[0] << k for k in range(1, 10)]
        bucket = np.searchsorted(t, deg, side="left")
        order = np.argsort(-bucket, kind="stable")
    else:
        order = np.argsort(deg, kind="stable")[::-1]
    new = np.empty(V, np.uint32)
    new[order] = np.arange(V, dtype=np.uint32)
    np.testing.assert_array_equal(el.label_array, new)
    np.testing.assert_array_equal(el.src, new[src])
    np.testing.assert_array_equal(el.dst, new[dst])
