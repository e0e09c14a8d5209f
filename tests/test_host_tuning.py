"""The SAP block kernel's launch variant is chosen for the size of the launch,
with the library's host code run over a stand-in for the CUDA runtime: a
variant that is fastest with one CTA per SM at most is not used by a batch of
systems that makes more, and a fixed variant is used by both."""
import ctypes as C

import pytest

import hostlib

BS = (4, 4, 4, 4)
ONE = b"Li256ELi1E"      # one site per lane pair, 256 threads, one CTA per SM


@pytest.fixture()
def qb():
    qb = hostlib.load()
    qb.lib().fake_fast.argtypes = [C.c_char_p, C.c_int]
    return qb


def _batch(qb, L, nr):
    """a function that runs a batch of n systems and returns its launches of the
    variant above, after a first batch of nr"""
    qb.geometry(L, BS, qb.even_first_ipt(L))
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.3, 1)
    qb.sw_term()
    qb.set_sap_parms(BS, 1, 4, 2)
    qb.set_cuda_graphs(0)
    f = qb.lib()

    def run(n):
        E, P = ([qb.DevField(64) for _ in range(n)] for _ in range(2))
        before = f.fake_launched(ONE)
        qb.dev_gcr_batch(2, 2, 0, 1e-10, [0.0] * n, E, P)
        return f.fake_launched(ONE) - before
    run(nr)
    return run


@pytest.mark.parametrize("L,nr,many", [((8, 8, 8, 8), 8, False), ((16, 16, 16, 16), 4, True), ((16, 16, 16, 16), 1, False),
                                       ((32, 16, 16, 16), 1, True)])
@pytest.mark.parametrize("graphs", [0, 1])
def test_choice_by_launch_size(qb, L, nr, many, graphs):
    qb.lib().fake_fast(ONE, 148)
    run = _batch(qb, L, nr)
    if graphs:
        qb.set_cuda_graphs(1)      # several systems in one launch need them
        run(nr)
        qb.set_cuda_graphs(0)
        qb.set_cuda_graphs(1)      # captured anew
    used = run(nr)
    if nr > 1 and not graphs:
        many = False               # one launch per system
    if L == (32, 16, 16, 16):
        many = True
    assert (used == 0) == many
    v = qb.sap_tuning(12)[0]
    assert (v == 1) == (L != (32, 16, 16, 16))
    qb.set_sap_variant(1)
    qb.set_cuda_graphs(0)
    qb.set_cuda_graphs(graphs)
    assert run(nr) > 0


# sites per parity of the blocks, variants that do not fit them
REFUSED = [((4, 4, 4, 4), []), ((4, 4, 8, 4), [5]), ((4, 4, 6, 6), [0, 5]), ((4, 8, 4, 6), [0, 4, 5]),
           ((6, 6, 6, 6), [0, 4, 5]), ((8, 8, 4, 6), [0, 4, 5])]


@pytest.mark.parametrize("bs,refused", REFUSED, ids=["x".join(map(str, b)) for b, _ in REFUSED])
def test_fixed_variants(qb, bs, refused):
    """the numbers that were good for a block size are: 0 up to 256 sites per
    parity, 1 to 3 for every size"""
    L = tuple(2 * b for b in bs)
    qb.geometry(L, bs, qb.even_first_ipt(L))
    qb.set_parms(1.5, 0.0, 0)
    qb.random_ud(0.3, 1)
    qb.sw_term()
    qb.set_sap_parms(bs, 1, 4, 2)
    x = [qb.DevField(32) for _ in range(2)]
    for v in range(6):
        if v in refused:
            with pytest.raises(qb.B200Error):
                qb.set_sap_variant(v)
            continue
        qb.set_sap_variant(v)
        qb.dev_sap(0.0, 1, 4, 1, *x)
        assert qb.sap_tuning(12)[1] >= 32 * ((bs[0] * bs[1] * bs[2] * bs[3] // 2 + 47) // 48)
    with pytest.raises(qb.B200Error):
        qb.set_sap_variant(6)
