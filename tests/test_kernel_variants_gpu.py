"""Every variant of the product kernels at the sizes where it can go wrong, against a plain loop over k.

Minima, maxima, words and whole-number sums do not depend on an order, so everything is compared for equality."""
import numpy as np
import pytest

from cuasr_b200 import Arguments, DType, Layout, Op, RINGS, Srgemm, Status, device_status, identity, srgemm_path
from cuasr_b200 import apsp

pytestmark = pytest.mark.gpu
COL, ROW = Layout.COLUMN_MAJOR, Layout.ROW_MAJOR
DTYPE = {"f32": DType.F32, "f64": DType.F64, "s32": DType.S32, "u32": DType.U32}


def torch_type(dtype):
    import torch
    return {"f32": torch.float32, "f64": torch.float64}.get(dtype, torch.int32)


def stored(x, layout, pad):
    """(flat storage of the matrix x in `layout` with `pad` unused elements per line, leading dimension)."""
    import torch
    lines = x if layout == ROW else x.T
    buf = torch.full((lines.shape[0], lines.shape[1] + pad), 77, dtype=x.dtype, device=x.device)
    buf[:, :lines.shape[1]] = lines
    return buf.reshape(-1), lines.shape[1] + pad


def read(flat, layout, m, n, ld):
    return flat.reshape(-1, ld)[:, :n] if layout == ROW else flat.reshape(-1, ld)[:, :m].T


def by_loop(ring, A, B, C):
    """(+) over k, then (+) C, one k at a time; as the library documents it, a NaN product is never taken and a NaN in
    C stays."""
    import torch
    add = {"minimum": torch.fmin, "maximum": torch.fmax, "plus": torch.add, "bit_xor": torch.bitwise_xor,
           "binary_or": torch.logical_or}
    mul = {"plus": torch.add, "minimum": torch.minimum, "maximum": torch.maximum, "multiplies": torch.mul,
           "bit_and": torch.bitwise_and, "binary_and": torch.logical_and}
    a, b = next((x, ring[len(x) + 1:]) for x in add if ring.startswith(x + "_"))
    if b.startswith("binary") or a.startswith("binary"):
        A, B, C = A != 0, B != 0, C != 0
    acc = mul[b](A[:, :1], B[:1, :])
    for k in range(1, A.shape[1]):
        acc = add[a](acc, mul[b](A[:, k:k + 1], B[k:k + 1, :]))
    if C.is_floating_point() and a in ("minimum", "maximum"):
        return torch.where(C.isnan(), C, add[a](acc, C))
    return add[a](acc, C)


def check_product(ring, dtype, A, B, C, layouts, pads=(0, 0, 0), workspace=False, mul_identity=None, in_place=False,
                  beta=None, screened=None):
    """screened: on the screened kernel, in that many pieces (0: chosen by size).  Returns the route."""
    import torch
    (m, k), n = A.shape, B.shape[1]
    add, mul = RINGS[ring]
    true_inf = dtype in ("f32", "f64")
    one = identity(mul, DTYPE[dtype], true_infinity=true_inf)
    op = Srgemm(add, mul, DTYPE[dtype], *layouts, add_identity=identity(add, DTYPE[dtype], true_infinity=true_inf),
                **({} if mul_identity is None else {"mul_identity": mul_identity}))
    (fa, lda), (fb, ldb), (fc, ldc) = (stored(x, lay, p) for x, lay, p in zip((A, B, C), layouts, pads))
    fd = fc if in_place else torch.full_like(fc, 77)
    args = Arguments((m, n, k), (fa, lda), (fb, ldb), (fc, ldc), (fd, ldc), (one, one if beta is None else beta))
    need = op.get_optional_workspace_size(args) if workspace else 0
    ws = torch.empty(need, dtype=torch.uint8, device="cuda") if need else None
    assert (op(args, ws) if screened is None else op.run_screened(args, screened, ws)) == Status.kSuccess
    got, want = read(fd, layouts[2], m, n, ldc), by_loop(ring, A, B, C if beta is None else C + beta)
    bad = ~((got == want) | ((got != got) & (want != want)))
    assert not bad.any(), (int(bad.sum()), bad.nonzero()[0].tolist(), got[bad][:3].tolist(), want[bad][:3].tolist())
    # nothing beyond the matrix was written
    lines = fd.reshape(-1, ldc)
    assert (lines[:, m if layouts[2] == COL else n:] == 77).all()
    return op.last_route()


def whole_numbers(g, shape, dtype, lo=-9, hi=10):
    import torch
    return torch.randint(0 if dtype == "u32" else lo, hi, shape, generator=g, device="cuda").to(torch_type(dtype))


# sizes at the edges of the 64 x 32, 64 x 64, 128 x 64 and 128 x 128 tiles and of their K steps, with few enough tiles
# that clusters of 2, 4 and 8 share K, and with enough that they do not
@pytest.mark.parametrize("ring, dtype", [("minimum_plus", "f32"), ("maximum_minimum", "f32"), ("plus_multiplies", "f64"),
                                         ("minimum_plus", "s32"), ("maximum_minimum", "s32"), ("minimum_plus", "u32"),
                                         ("bit_xor_bit_and", "u32"), ("binary_or_binary_and", "f32"), ("binary_or_binary_and", "f64"),
                                         ("binary_or_binary_and", "s32")])
@pytest.mark.parametrize("m, n, k", [(1, 1, 1), (33, 65, 31), (64, 32, 257), (63, 31, 1025), (65, 129, 513), (256, 192, 700),
                                     (300, 500, 129), (640, 1024, 100), (1025, 1100, 70)])
def test_tiles_and_clusters(cuda_device, ring, dtype, m, n, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m * 7 + n * 3 + k)
    A, B, C = (whole_numbers(g, s, dtype) for s in ((m, k), (k, n), (m, n)))
    for i, layouts in enumerate(((COL, COL, COL), (ROW, COL, ROW), (ROW, ROW, COL), (COL, ROW, ROW))):
        for pads in ((0, 0, 0), (1, 3, 2), ((-k) % 4, (-k) % 4, (-n) % 4)):
            check_product(ring, dtype, A, B, C, layouts, pads, workspace=i % 2 == 1)
    assert device_status() == 0


@pytest.mark.parametrize("dtype", ["f32", "f64", "s32"])
def test_logical_ring_of_any_value(cuda_device, dtype):
    """Everything but zero counts as true, negative zeros do not and NaN does; the result is 0 or 1 whatever the accumulation
    starts from."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(8)
    m, n, k = 130, 70, 67
    A, B = (torch.where(torch.rand(s, generator=g, device="cuda") < 0.1, whole_numbers(g, s, "s32", -3, 4), 0).to(torch_type(dtype))
            for s in ((m, k), (k, n)))
    if dtype != "s32":
        A, B = -A, torch.where(B == 1, torch.nan, torch.where(B == 2, torch.inf, torch.where(B == 3, 1e-42, B)))
    want = ((A != 0).double() @ (B != 0).double()) != 0
    assert want.any() and not want.all()
    add, mul = RINGS["binary_or_binary_and"]
    for start in (0, 1, 5):
        D = torch.full((m, n), 77, dtype=torch_type(dtype), device="cuda")
        op = Srgemm(add, mul, DTYPE[dtype], ROW, ROW, ROW, add_identity=start, mul_identity=1)
        args = Arguments((m, n, k), (A, k), (B, n), (torch.zeros_like(D), n), (D, n), (1, 0))
        assert op(args) == Status.kSuccess
        assert (D == (want | (start != 0)).to(D.dtype)).all(), start


# pieces of every tile, and whole tiles in front of pieces of the last wave's
@pytest.mark.parametrize("ring, dtype, m, n, k", [("minimum_plus", "f32", 1500, 1000, 2048), ("maximum_plus", "f64", 1500, 1000, 1024),
                                                  ("plus_multiplies", "f64", 1500, 2048, 2048), ("maximum_minimum", "s32", 1500, 1000, 2048),
                                                  ("maximum_minimum", "s32", 1500, 2048, 1024)])
def test_pieces_meet_through_tickets(cuda_device, ring, dtype, m, n, k):
    """The optional workspace of a launch that the model cuts along K; twice on the same workspace, whose contents do not matter
    and whose tickets the first launch has used."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(k)
    A, B, C = (whole_numbers(g, s, dtype) for s in ((m, k), (k, n), (m, n)))
    want = by_loop(ring, A, B, C)
    add, mul = RINGS[ring]
    true_inf = dtype in ("f32", "f64")
    one = identity(mul, DTYPE[dtype], true_infinity=true_inf)
    op = Srgemm(add, mul, DTYPE[dtype], ROW, COL, ROW, add_identity=identity(add, DTYPE[dtype], true_infinity=true_inf))
    B = B.T.contiguous()
    ws = None
    for _ in range(2):
        D = torch.full_like(C, 77)
        args = Arguments((m, n, k), (A, k), (B, k), (C, n), (D, n), (one, one))
        if ws is None:
            ws = torch.full((op.get_optional_workspace_size(args),), 0x5A, dtype=torch.uint8, device="cuda")
        assert op(args, ws) == Status.kSuccess
        assert "tickets=1" in op.last_route(), op.last_route()
        assert (D == want).all()
    assert device_status() == 0


def test_ragged_k_does_not_lean_on_the_identities(cuda_device):
    """An integer minimum has no neutral padding: a K that ends inside a K step must not bring in products of the
    caller's identities, whatever they are."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    for m, n, k in ((40, 50, 7), (200, 150, 45), (256, 192, 77)):
        A, B = (whole_numbers(g, s, "s32", 100, 200) for s in ((m, k), (k, n)))
        C = torch.full((m, n), 1000, dtype=torch.int32, device="cuda")
        for layouts in ((COL, COL, COL), (ROW, COL, ROW)):
            check_product("minimum_plus", "s32", A, B, C, layouts, (1, 1, 0), mul_identity=-2**31)
            route = check_product("minimum_plus", "s32", A, B, C, layouts, (1, 1, 0), True, mul_identity=-2**31)
            assert ("a=copy+tma b=copy+tma" in route) == (m == 256), route


# ---- double precision minima and maxima, screened in 16 bits -------------------------------------------------------
def distances(kind, g, shape, along):
    """Values of a product of double precision tropical matrices; `along`: the axis that is contracted."""
    import torch
    dev = "cuda"
    x = torch.rand(shape, generator=g, device=dev, dtype=torch.float64)
    if kind == "edges":              # a sparse weighted graph
        return torch.where(torch.rand(shape, generator=g, device=dev) < 0.1, 1 + 999 * x, torch.inf)
    if kind == "signed":
        return 200 * x - 100
    if kind == "ties":
        return torch.randint(0, 3, shape, generator=g, device=dev).double()
    if kind == "falling":            # every k improves every element
        steps = torch.arange(shape[along], 0, -1, device=dev, dtype=torch.float64)
        return x * 0.01 + (steps[None, :] if along == 1 else steps[:, None])
    if kind == "wide":               # magnitudes that fit neither 16 bits nor fp32
        return 10.0 ** (x * 600 - 300)
    if kind == "almost zero":        # negative values and differences far below the resolution of the largest one
        small = torch.randint(-3, 4, shape, generator=g, device=dev).double() * 1e-310
        return torch.where(x < 0.01, 3e38, torch.where(x < 0.5, 0.0, small))
    if kind == "bursts":             # stretches of k with negative values between ones that fit the screen: exact runs of
        k = torch.arange(shape[along], device=dev)        # blocks, screened blocks behind them
        burst = ((k // 32) % 7 < 3) & (k % 32 == 5)
        return torch.where(burst[None, :] if along == 1 else burst[:, None], 90 - 100 * x, 100 * x + 1)
    if kind == "nan":
        return torch.where(x < 0.002, torch.nan, torch.where(x < 0.3, torch.inf, 100 * x))
    return torch.where(x < 0.002, -torch.inf, 100 * x)


KINDS = ["edges", "signed", "ties", "falling", "wide", "almost zero", "bursts", "nan", "infinite"]


def tropical_operands(ring, kind, m, n, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(k)
    A, B = distances(kind, g, (m, k), 1), distances(kind, g, (k, n), 0)
    C = distances(kind, g, (m, n), 0)
    if ring == "maximum_plus" and kind in ("edges", "nan", "falling"):
        A, B, C = (torch.where(x == torch.inf, -torch.inf, x) for x in (A, B, C))
        if kind == "falling":
            A, B = A.flip(1), B.flip(0)
    if ring == "maximum_plus" and kind == "infinite":
        A, B = (torch.where(x == -torch.inf, torch.inf, x) for x in (A, B))
    return A, B, C


# the screened kernel whatever the data: one piece of K per tile of the output, and several (which then meet in D), one of them of a
# single block; even and odd lines, every tile and K edge
@pytest.mark.parametrize("m, n, k, pieces", [(700, 650, 1500, 1), (1021, 1023, 517, 3), (129, 1290, 2000, 5), (64, 70, 5001, 157),
                                             (2305, 1025, 650, 1), (1, 3, 33, 2), (300, 129, 32, 1)])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("ring", ["minimum_plus", "maximum_plus"])
def test_screened_kernel(cuda_device, ring, kind, m, n, k, pieces):
    import torch
    A, B, C = tropical_operands(ring, kind, m, n, k)
    for layouts, pads, C, in_place in (((ROW, COL, ROW), (-k % 2, -k % 2, 0), C, False), ((COL, COL, COL), (1, 0, 1), C, True),
                                       ((COL, ROW, ROW), (0, 0, 0), torch.full_like(C, -5.0 if ring == "minimum_plus" else 1e12), False)):
        route = check_product(ring, "f64", A, B, C, layouts, pads, in_place=in_place, screened=pieces)
        assert route.startswith("screened tile=128x128") and f"pieces={pieces} " in route, route
    assert device_status() == 0


# Sizes at which both kernels are launched and the operands decide which of them does the product: in several pieces that meet in D
# and in one; and a size that always runs exactly.  With D in place of C and a factor on it, a product done twice shows.
@pytest.mark.parametrize("m, n, k, pieces", [(1000, 1000, 3000, 2), (1021, 1023, 4099, 2), (400, 390, 12001, 9), (2049, 2047, 2050, 1),
                                             (500, 520, 600, 0)])
@pytest.mark.parametrize("kind", KINDS + ["rare"])
@pytest.mark.parametrize("ring", ["minimum_plus", "maximum_plus"])
def test_screened_or_exact(cuda_device, ring, kind, m, n, k, pieces):
    import torch
    A, B, C = tropical_operands(ring, "ties" if kind == "rare" else kind, m, n, k)
    if kind == "rare":               # values the screen cannot hold, few enough for the sample to miss some
        g = torch.Generator(device="cuda").manual_seed(n)
        A, B = (torch.where(torch.rand(x.shape, generator=g, device="cuda") < 2e-4, -x - 1, x) for x in (A, B))
    for layouts, pads, in_place, workspace in (((ROW, COL, ROW), (-k % 2, -k % 2, 0), False, False), ((COL, COL, COL), (1, 0, 1), True, True),
                                               ((COL, ROW, ROW), (0, 0, 0), True, False)):
        route = check_product(ring, "f64", A, B, C, layouts, pads, workspace, in_place=in_place, beta=3.0)
        assert ("or product" in route) == (pieces > 0) and (pieces == 0 or route.startswith(f"screened pieces={pieces} ")), route
    assert device_status() == 0


@pytest.mark.parametrize("ring", ["minimum_plus", "maximum_plus"])
@pytest.mark.parametrize("m, n, k", [(1000, 1000, 3000), (2049, 2047, 2050), (300, 200, 100)])
def test_double_precision_tropical_zeros_are_positive(cuda_device, ring, m, n, k):
    """D = (0 + A B) (+) (0 + C): adding zero makes every zero a positive one, whichever kernel does it."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(m)
    sign = -1.0 if ring == "minimum_plus" else 1.0
    better = Op.MINIMUM if ring == "minimum_plus" else Op.MAXIMUM
    A, B = (torch.where(torch.rand(s, generator=g, device="cuda") < 0.001, -0.0, -sign) for s in ((m, k), (k, n)))
    A, B = A.double(), B.double()
    if ring == "maximum_plus":
        A, B = -A.abs(), -B.abs()                 # best sums: -0 + -0
    for beta in (0.0, -0.0):
        C = torch.full((m, n), -sign * 5, dtype=torch.float64, device="cuda")
        C[::2] = -0.0
        D = torch.empty_like(C)
        op = Srgemm(better, Op.PLUS, DType.F64, ROW, ROW, ROW, add_identity=-sign * np.inf)
        assert op(Arguments((m, n, k), (A, k), (B, n), (C, n), (D, n), (0.0, beta))) == Status.kSuccess
        zero = D == 0
        assert zero.any() and (zero == (by_loop(ring, A, B, C) == 0)).all()
        if beta == 0.0 and not np.signbit(beta):
            assert not torch.signbit(D[zero]).any(), (int(torch.signbit(D[zero]).sum()), op.last_route())
        else:
            assert op.last_route().startswith("product ")
            continue
        args = Arguments((m, n, k), (A, k), (B, n), (C, n), (D, n), (0.0, beta))
        assert op.run_screened(args) == Status.kSuccess
        assert ((D == 0) == zero).all() and not torch.signbit(D[zero]).any()


def test_double_precision_tropical_product_into_host_memory(cuda_device):
    """A D in mapped host memory is written once, by the exact kernel; under capture the question where D lies is asked too."""
    import torch
    m, n, k = 1000, 1000, 3000
    g = torch.Generator(device="cuda").manual_seed(2)
    A, B = (torch.rand(s, generator=g, device="cuda", dtype=torch.float64) for s in ((m, k), (k, n)))
    C = torch.full((m, n), torch.inf, dtype=torch.float64, device="cuda")
    host = torch.zeros((m, n), dtype=torch.float64).pin_memory()
    here, captured = torch.zeros_like(C), torch.zeros_like(C)
    op = Srgemm(Op.MINIMUM, Op.PLUS, DType.F64, ROW, ROW, ROW, add_identity=np.inf)

    def product(D):
        args = Arguments((m, n, k), (A, k), (B, n), (C, n), (D, n), (0.0, 0.0))
        assert op(args, None, torch.cuda.current_stream()) == Status.kSuccess
        return op.last_route()
    assert product(host).startswith("product ")
    assert product(here).startswith("screened pieces=2 or product ")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert product(captured).startswith("screened pieces=2 or product ")
    graph.replay()
    torch.cuda.synchronize()
    want = by_loop("minimum_plus", A, B, C)
    assert (here == want).all() and (captured == want).all() and (host.cuda() == want).all()
    assert device_status() == 0


# ---- distances with predecessors ----------------------------------------------------------------------------------
# the 128 x 128 tile, and the 64 x 64 one with K shared by the CTAs of clusters
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("m, n, k", [(1, 1, 1), (64, 64, 65), (65, 63, 200), (130, 190, 700), (300, 200, 1030), (1500, 1400, 90)])
def test_path_kernel_variants(cuda_device, dtype, m, n, k):
    import torch
    g = torch.Generator(device="cuda").manual_seed(k)
    for maximize in (False, True):
        for kind in ("ties", "falling", "nan"):
            A, B = (distances(kind, g, s, a).to(torch_type(dtype)) for s, a in (((m, k), 1), ((k, n), 0)))
            dist = torch.full((m, n), -1.0 if maximize else 2.0, dtype=A.dtype, device="cuda")
            dist[::3] = -torch.inf if maximize else torch.inf
            if kind == "nan":
                dist[:, ::5] = torch.nan
            parent = torch.full((m, n), -7, dtype=torch.int32, device="cuda")
            want, via = dist.clone(), parent.clone()
            for q in range(k):
                s = A[:, q:q + 1] + B[q:q + 1, :]
                better = s > want if maximize else s < want
                want, via = torch.where(better, s, want), torch.where(better, q + 5, via)
            for layouts, pads in (((COL, COL, COL), (1, 0, 2)), ((ROW, COL, ROW), (-k % 4, -k % 4, 0))):
                (fa, lda), (fb, ldb), (fd, ldd), (fp, ldp) = (stored(x, lay, p) for x, lay, p in zip(
                    (A, B, dist, parent), layouts + layouts[2:], pads + (1,)))
                op = Srgemm(Op.MAXIMUM if maximize else Op.MINIMUM, Op.PLUS, DTYPE[dtype], *layouts)
                assert srgemm_path(op, (m, n, k), (fa, lda), (fb, ldb), (fd, ldd), (fp, ldp), k_offset=5) == Status.kSuccess
                got = read(fd, layouts[2], m, n, ldd)
                assert ((got == want) | (got.isnan() & want.isnan())).all(), (maximize, kind, layouts)
                assert (read(fp, layouts[2], m, n, ldp) == via).all(), (maximize, kind, layouts)
    assert device_status() == 0


# ---- the closure of diagonal blocks -------------------------------------------------------------------------------
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n, block", [(1, 0), (2, 0), (63, 0), (65, 0), (127, 0), (128, 0), (129, 0), (300, 0), (300, 100),
                                      (300, 260), (700, 640)])
def test_closure_of_diagonal_blocks(cuda_device, dtype, n, block):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    w = torch.randint(1, 50, (n, n), generator=g, device="cuda").to(torch_type(dtype))
    # distances from 10 * v up when going to a later vertex v, down when coming back: negative edges, no negative cycle
    height = 10 * torch.arange(n, device="cuda").to(w.dtype)
    w += height[None, :] - height[:, None]
    w[torch.rand((n, n), generator=g, device="cuda") > min(1.0, 6.0 / n)] = torch.inf
    w.fill_diagonal_(0)
    want = w.clone()
    for k in range(n):
        want = torch.minimum(want, want[:, k:k + 1] + want[k:k + 1, :])
    flat, ld = stored(w, COL, 3)
    assert apsp.device_solve(flat, n, DTYPE[dtype], apsp.BLOCKED_FLOYD_WARSHALL, ldd=ld, block=block) == Status.kSuccess
    assert (read(flat, COL, n, n, ld) == want).all()
    assert device_status() == 0


# ---- launches that overlap the end of the one before --------------------------------------------------------------
def test_dependent_launches_on_streams_and_under_capture(cuda_device):
    """Each product reads the result of the one before it, with copies in between and a second stream joined in."""
    import torch
    n, g = 96, torch.Generator(device="cuda").manual_seed(3)
    start = torch.randint(0, 50, (n, n), generator=g, device="cuda").float()
    op = Srgemm(Op.MINIMUM, Op.PLUS, DType.F32, COL, COL, COL, add_identity=np.float32(np.inf))
    x, y, z, w = (torch.empty(n * n, device="cuda") for _ in range(4))

    def product(a, b, c, stream):
        assert op(Arguments((n, n, n), (a, n), (b, n), (c, n), (c, n), (0.0, 0.0)), None, stream) == Status.kSuccess

    def work():
        s, other = torch.cuda.current_stream(), side
        x.copy_(start.reshape(-1)); y.copy_(x); z.fill_(torch.inf); w.copy_(x)
        product(x, x, y, s)
        product(y, y, x, s)
        other.wait_stream(s)
        product(x, y, z, other)
        product(x, y, w, s)                 # beside the one before
        s.wait_stream(other)
        product(w, z, x, s)
        return x

    side = torch.cuda.Stream()
    main = torch.cuda.Stream()
    with torch.cuda.stream(main):
        work()
    main.synchronize()
    plain = x.clone()

    def loop(a, b, c):                          # column-major storage: the transposed matrices
        out = c
        for k in range(n):
            out = torch.minimum(out, a[:, k:k + 1] + b[k:k + 1, :])
        return out
    X, W, Z = start.T, start.T, torch.full((n, n), torch.inf, device="cuda")
    Y = loop(X, X, X)
    X = loop(Y, Y, X)
    Z = loop(X, Y, Z)
    W = loop(X, Y, W)
    X = loop(W, Z, X)
    assert (plain.reshape(n, n).T == X).all()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=main):
        work()
    for _ in range(3):
        x.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert (x == plain).all()
    assert device_status() == 0
