"""GPU parity of the operator kernels' newer paths against the oracle's H*v (the reference restated in FP64).

Tolerances: a row sums at most a few hundred products of FP64 values, so FP64 results agree to about 1e-13 of the
largest element; FP32 vectors carry their 6e-8 rounding per term, 2e-6 in all.
"""
import numpy as np
import pytest

from edlib_gb300 import models

pytestmark = pytest.mark.gpu

TOL = {"fp64": 1e-13, "fp32": 2e-6}


@pytest.fixture(scope="module")
def ed():
    from edlib_gb300 import build
    build.build()
    from edlib_gb300 import ed as _ed
    _ed.context(0)
    return _ed


def check_products(ed, params, data, kind, storage, sectors, precision, seed=3, scale_rows=None):
    from oracle.oracle import OracleED
    params = dict(params)
    params.update({"storage.MAX_DIM": 0, "storage.MAX_SIZE": 0})
    ham = ed.Hamiltonian(params, data, storage=storage, precision=precision)
    ham.set_limits(0, 0)
    o = OracleED(params, data, storage, kind)
    rng = np.random.default_rng(seed)
    for sec in sectors:
        n = ham.storage.fill(*sec)
        assert o.fill(*sec) == n
        v = rng.standard_normal(n)
        w = o.av(v)
        tol = TOL[precision] * np.abs(w).max()
        assert np.abs(ham.storage.av(v) - w).max() <= tol, (storage, sec)
        assert np.abs(ham.storage.av(v, w=np.ones(n), clear=False) - (w + 1.0)).max() <= tol + TOL[precision], (storage, sec)
    ham.close()


def general_siam(ns, ml, seed):
    """An impurity whose interaction tensor has every term (real symmetric H): terms between the spins with a hop
    or an occupation on either side, and two-body hops inside one spin."""
    rng = np.random.default_rng(seed)
    nk = ns - ml
    eps = rng.uniform(-1, 1, nk)
    v = rng.uniform(-0.5, 0.5, (ml, nk))
    T = rng.uniform(-1, 1, (ml,) * 4)
    T = T + T.transpose(1, 0, 3, 2)          # the two halves of a term exchanged
    T = T + T.transpose(2, 3, 0, 1)          # its transpose
    h0 = np.zeros((ml, ml, 2))
    data = models.siam(np.stack([eps, eps], 1), np.stack([v, v], -1), h0, 0.3, T)
    return {"NSITES": ns, "NSPINS": 2, "siam.NORBITALS": ml}, data


# rows of 1 to 70 states (flat), 252 (16-byte tiles), 495 (lane-strided tiles); a full tensor and a Kanamori one
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("model,ns,sectors", [
    ("general", 5, [(0, 3), (2, 3), (5, 1), (4, 5)]), ("general", 8, [(4, 4), (3, 6)]), ("general", 10, [(3, 5), (5, 6)]),
    ("kanamori", 7, [(3, 3), (4, 2)]), ("kanamori", 12, [(2, 6), (3, 4)])])
def test_interaction_products_against_oracle(ed, precision, model, ns, sectors):
    if model == "general":
        params, data = general_siam(ns, 3, ns)
    else:
        params, data = models.random_kanamori_siam(ns, nbath_per_orb=[(ns - 3 + 2 - m) // 3 for m in range(3)])
    check_products(ed, params, data, "SIAM", "SRS", sectors, precision)


# edges of the row-interleaved tiles: rows of 128 to 2047 states, a multiple of four or not, last tiles of few columns,
# items whose last group has one to three rows, single-row sectors, rows just inside and outside the range
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ns,sectors", [
    (10, [(0, 5), (1, 4), (2, 5), (10, 6)]), (11, [(1, 4), (9, 3), (2, 5)]), (12, [(3, 4), (11, 6), (2, 3), (1, 8)]),
    (13, [(1, 5), (2, 6), (12, 7)]), (14, [(1, 4), (13, 5)])])
def test_row_interleaved_tiles_against_oracle(ed, precision, ns, sectors):
    params, data = models.random_siam(40 + ns, ns - 1)
    check_products(ed, params, data, "SIAM", "SRS", sectors, precision)
    t = models.ring_hopping(ns, 1.0)
    t[0, ns // 2] = t[ns // 2, 0] = 0.4
    check_products(ed, {"NSITES": ns, "NSPINS": 2}, models.hubbard(t, 3.0, 1.0), "HUBBARD", "SRS", sectors[:2], precision)


def test_device_vectors_off_16_byte_bases(ed):
    """edgpu_spmv on vectors that start 4 (FP32) or 8 (FP64) bytes past a 16-byte boundary, and with an odd distance:
    the same values as on aligned ones, to the last bit."""
    import torch
    from edlib_gb300 import _abi
    params, data = models.random_siam(5, 11)
    ham = ed.Hamiltonian(ed.Params(params), data, storage="SRS", precision="fp64")
    ham.set_limits(0, 0)
    L = _abi.lib()
    for sec in ((2, 6), (3, 4)):
        n = ham.storage.fill(*sec)
        for prec, dt in ((0, torch.float64), (1, torch.float32)):
            x = torch.randn(2, n, dtype=dt, device="cuda")
            ys = []
            for off, ld in ((0, (n + 3) // 4 * 4), (1, n + 1 + n % 2)):
                bx = torch.zeros(2 * ld + 8, dtype=dt, device="cuda")
                by = torch.zeros(2 * ld + 8, dtype=dt, device="cuda")
                for q in range(2):
                    bx[off + q * ld:off + q * ld + n] = x[q]
                torch.cuda.synchronize()
                rc = L.edgpu_spmv(ham._m, 1, sec[0], sec[1], bx[off:].data_ptr(), by[off:].data_ptr(), 2, ld, prec, 0,
                                  torch.cuda.current_stream().cuda_stream)
                assert rc == 0
                torch.cuda.synchronize()
                ys.append(torch.stack([by[off + q * ld:off + q * ld + n] for q in range(2)]))
                assert by[:off].abs().sum() == 0 and by[off + 2 * ld:].abs().sum() == 0
            assert torch.equal(ys[0], ys[1]), (sec, prec)
    ham.close()


# rows of thousands of states: tiles of one group of rows; from 4096 states on two passes (512 up rows or more; odd and
# even row lengths) or one row at a time (fewer)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_rows_of_thousands_of_states_against_oracle(ed, precision):
    n = 14
    t = models.ring_hopping(n, 1.0)
    t[0, 5] = t[5, 0] = -0.3
    check_products(ed, {"NSITES": n, "NSPINS": 2}, models.hubbard(t, 4.0, 2.0), "HUBBARD", "SRS",
                   [(4, 6), (4, 7), (3, 7), (2, 6)], precision)
    params, data = models.random_kanamori_siam(3, [4, 4, 3])
    check_products(ed, params, data, "SIAM", "SRS", [(4, 8), (1, 7)], precision)
    params, data = models.random_kanamori_siam(4, [4, 4, 4])  # 15 orbitals: rows of 5005 and 6435 states
    check_products(ed, params, data, "SIAM", "SRS", [(11, 6), (4, 7), (1, 8), (2, 9)], precision)


def test_first_product_on_a_callers_stream_sees_complete_tables(ed):
    """edgpu_spmv on a stream of the caller's right after the sector's tables were enqueued on the context's own
    stream: the same values as a call made when everything has finished."""
    import torch
    from edlib_gb300 import _abi
    L = _abi.lib()
    s = torch.cuda.Stream()
    for seed in range(6):
        params, data = models.random_siam(seed, 11)
        ham = ed.Hamiltonian(ed.Params(params), data, storage="SRS", precision="fp64")
        ham.set_limits(0, 0)
        for sec in ((6, 3), (2, 6), (6, 1)):
            n = ham.vector_size(sec)
            x = torch.randn(n, dtype=torch.float64, device="cuda")
            y = [torch.zeros_like(x) for _ in range(2)]
            torch.cuda.synchronize()
            for q in range(2):
                assert L.edgpu_spmv(ham._m, 1, sec[0], sec[1], x.data_ptr(), y[q].data_ptr(), 1, n, 0, 0, s.cuda_stream) == 0
                torch.cuda.synchronize()
            assert torch.equal(y[0], y[1]), (seed, sec)
        ham.close()


# CRS and SOCRS rows shared by several lanes: fewer rows than lanes, item remainders, all transition kinds
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("storage", ["CRS", "SOCRS"])
def test_row_storages_against_oracle(ed, storage, precision):
    t = models.square_hopping(2, 4, 1.0, -0.2)
    check_products(ed, {"NSITES": 8, "NSPINS": 2}, models.hubbard(t, 3.0, 1.5, hmag=0.05), "HUBBARD", storage,
                   [(0, 0), (0, 1), (1, 1), (1, 7), (2, 3), (4, 4)], precision)
    params, data = models.random_siam(11, 9)
    check_products(ed, params, data, "SIAM", storage, [(10, 9), (5, 3), (5, 5)], precision)
    # interaction terms of one spin order: SOCRS refuses the two that meet in one element
    params, data = models.random_kanamori_siam(2, [2, 1, 2])
    data["interaction/values"] = data["interaction/values"].copy()
    data["interaction/values"][1] = 0.0
    data["interaction/values"][0, 0] = 0.0
    check_products(ed, params, data, "SIAM", storage, [(1, 2), (4, 3)], precision)
    if storage == "CRS":
        params, data = general_siam(6, 3, 5)
        check_products(ed, params, data, "SIAM", storage, [(3, 3), (2, 4)], precision)


# items of as few as four rows (one vector), the sector's own items (40 vectors): each element is summed in the same
# order, so its value does not depend on the split
@pytest.mark.parametrize("precision,storage,ns,sec", [
    ("fp32", "SRS", 12, (6, 6)), ("fp64", "SRS", 12, (5, 4)), ("fp32", "SRS", 10, (5, 2)), ("fp64", "SRS", 7, (3, 3)),
    ("fp64", "CRS", 8, (4, 4)), ("fp32", "SOCRS", 10, (5, 4))])
def test_device_products_independent_of_the_number_of_vectors(ed, precision, storage, ns, sec):
    import torch
    from edlib_gb300 import _abi
    params, data = models.random_siam(7, ns - 1)
    ham = ed.Hamiltonian(ed.Params(params), data, storage=storage, precision=precision)
    ham.set_limits(0, 0)
    n = ham.storage.fill(*sec)
    ld = (n + 3) // 4 * 4
    x = torch.randn(40, ld, dtype=torch.float64 if precision == "fp64" else torch.float32, device="cuda")
    for acc in (0, 1):
        ys = []
        for nvec in (1, 3, 40):
            y = torch.ones_like(x)
            rc = _abi.lib().edgpu_spmv(ham._m, _abi.STORAGES[storage], sec[0], sec[1], x.data_ptr(), y.data_ptr(), nvec, ld,
                                       _abi.PRECISIONS[precision], acc, torch.cuda.current_stream().cuda_stream)
            assert rc == 0
            torch.cuda.synchronize()
            assert bool((y[nvec:] == 1).all())
            ys.append(y[0, :n])
        assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])
    ham.close()


def test_recurrences_alone_and_in_a_batch_of_many_items(ed):
    """One model's recurrences have an item per block and start early behind one another; those of eight together have
    more items than blocks and ordinary launches.  Sums run in a fixed order in both: equal to the last bit."""
    specs = []
    for seed in range(8):
        p, d = models.random_siam(300 + seed, 9)
        p.update({"arpack.NEV": 2, "lanc.BETA": 20.0, "lanc.NOMEGA": 64, "lanc.NLANC": 40, "arpack.SECTOR": 1})
        d["sectors/values"] = np.array([(5, 5)], dtype=np.float64)
        specs.append((ed.Params(p), d))
    hams = [ed.Hamiltonian(p, d, storage="SRS", precision="fp64") for p, d in specs]
    for h in hams:
        h.set_limits(0, 0)
        h.diag()
    alone = [ed.GreensFunction(p, h).compute() for (p, _), h in zip(specs, hams)]
    Gs, _, _ = ed.greens_function_many(specs[0][0], hams)
    assert all(np.array_equal(a, b) for a, b in zip(alone, Gs))


# items that lie across the sector's own ones (12 -> 8 rows, 24 -> 20), with more up hops than any of those: the values
# of a call with many vectors to the last bit, and the oracle's
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("ns,sec,nvec", [(13, (6, 3), 1), (18, (4, 2), 2)])
def test_items_across_the_sectors_own_ones(ed, precision, ns, sec, nvec):
    import torch
    from edlib_gb300 import _abi
    from oracle.oracle import OracleED
    params, data = models.random_siam(70 + ns, ns - 1)
    params.update({"storage.MAX_DIM": 0, "storage.MAX_SIZE": 0})
    ham = ed.Hamiltonian(ed.Params(params), data, storage="SRS", precision=precision)
    ham.set_limits(0, 0)
    n = ham.storage.fill(*sec)
    ld = (n + 3) // 4 * 4
    x = torch.randn(40, ld, dtype=torch.float64 if precision == "fp64" else torch.float32, device="cuda")
    ys = []
    for k in (nvec, 40):
        y = torch.zeros_like(x)
        assert _abi.lib().edgpu_spmv(ham._m, 1, sec[0], sec[1], x.data_ptr(), y.data_ptr(), k, ld,
                                     _abi.PRECISIONS[precision], 0, torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        ys.append(y[:nvec, :n])
    assert torch.equal(ys[0], ys[1])
    o = OracleED(params, data, "SRS", "SIAM")
    assert o.fill(*sec) == n
    w = o.av(x[0, :n].double().cpu().numpy())
    assert np.abs(ys[0][0].double().cpu().numpy() - w).max() <= TOL[precision] * np.abs(w).max()
    ham.close()


# item sizes at both ends of EDGPU_SRS_ITEM_ELEMS (read once, so in a fresh process), on a cluster whose sites are all bound
# to one another: most up hops per item
@pytest.mark.parametrize("elems", [512, 24576])
def test_item_sizes_against_oracle(elems):
    import os
    import subprocess
    import sys
    code = (
        "import numpy as np\n"
        "from edlib_gb300 import ed, models\n"
        "from oracle.oracle import OracleED\n"
        "ed.context(0)\n"
        "rng = np.random.default_rng(9)\n"
        "t = rng.uniform(0.2, 1.0, (14, 14))\n"
        "t = t + t.T - np.diag(np.diag(t + t.T))\n"
        "params = {'NSITES': 14, 'NSPINS': 2, 'storage.MAX_DIM': 0, 'storage.MAX_SIZE': 0}\n"
        "data = models.hubbard(t, 3.0, 1.0)\n"
        "ham = ed.Hamiltonian(params, data, storage='SRS', precision='fp64')\n"
        "ham.set_limits(0, 0)\n"
        "o = OracleED(params, data, 'SRS', 'HUBBARD')\n"
        "for sec in [(7, 3), (6, 11)]:\n"
        "    n = ham.storage.fill(*sec)\n"
        "    assert o.fill(*sec) == n\n"
        "    v = rng.standard_normal(n)\n"
        "    w = o.av(v)\n"
        "    assert np.abs(ham.storage.av(v) - w).max() <= 1e-13 * np.abs(w).max(), sec\n"
        "    v /= np.linalg.norm(v)\n"
        "    a, b, _ = ed.lanczos(ham, sec, v, 3)\n"
        "    w = o.av(v)\n"
        "    assert abs(a[0, 0] - w @ v) <= 1e-12 and abs(b[0, 1] - np.linalg.norm(w - (w @ v) * v)) <= 1e-12, sec\n"
        "print('ok')\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, EDGPU_SRS_ITEM_ELEMS=str(elems), PYTHONPATH=root))
    assert r.returncode == 0 and "ok" in r.stdout, r.stderr[-3000:]


# an infinite element reaches its own place and those that H binds it to; every other element keeps its value (rows of
# 5005 states: two passes)
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_infinite_element_stays_on_its_bonds(ed, precision):
    params, data = models.random_siam(6, 14)
    ham = ed.Hamiltonian(ed.Params(params), data, storage="SRS", precision=precision)
    ham.set_limits(0, 0)
    n = ham.storage.fill(4, 6)
    v = np.random.default_rng(2).standard_normal(n)
    for i in (0, 5, n // 2 + 1234, n - 7):
        e, z, inf = np.zeros(n), v.copy(), v.copy()
        e[i], z[i], inf[i] = 1.0, 0.0, np.inf
        bound = ham.storage.av(e) != 0
        bound[i] = True
        w, w0 = ham.storage.av(inf), ham.storage.av(z)
        assert np.array_equal(w[~bound], w0[~bound])
    ham.close()


# short rows with many up hops (one element at a time; more hops per item than its shared memory holds) and few
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_short_rows_with_many_up_hops_against_oracle(ed, precision):
    t = models.square_hopping(4, 3, 1.0, -0.3)
    check_products(ed, {"NSITES": 12, "NSPINS": 2}, models.hubbard(t, 4.0, 2.0), "HUBBARD", "SRS", [(6, 1), (6, 2), (2, 10)],
                   precision)
    params, data = models.random_siam(3, 11)
    check_products(ed, params, data, "SIAM", "SRS", [(6, 1), (6, 2), (7, 0)], precision)


# float-float and FP64 recurrences one at a time (few items: launches that start early, two blocks per SM) and all in one
# batch: each path adds in the same order.  Items of one recurrence, and of the batch of four kept states' sixteen: 10
# orbitals 7 and 112, 11 29 and 400 (tiles, rows of 210 to 462 states); 9 orbitals 6 to 8 and 112 (rows of 126).
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("ns", [9, 10, 11])
def test_recurrences_independent_of_their_batch(ed, ns, precision):
    params, data = models.random_siam(21, ns - 1)
    params.update({"arpack.NEV": 4, "arpack.SECTOR": 1, "lanc.BETA": 2.0, "lanc.NOMEGA": 16, "lanc.NLANC": 60})
    data["sectors/values"] = np.array([[ns // 2, ns // 2]], dtype=np.float64)
    p = ed.Params(params)
    ham = ed.Hamiltonian(p, data, storage="SRS", precision=precision)
    ham.set_limits(0, 0)
    ham.diag()
    G = []
    for ham.max_batch in (0, 1, 3):
        g = ed.GreensFunction(p, ham)
        g.compute()
        G.append(g.G.copy())
    ham.close()
    assert np.all(np.isfinite(G[0])) and np.abs(G[0]).max() > 0
    assert np.array_equal(G[0], G[1]) and np.array_equal(G[0], G[2])
