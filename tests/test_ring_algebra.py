"""The ring terms of the doubles residual in two intermediates and two products (cc_ground.cpp)
against the reference's three and three (ccwfn.cc:400-430, :486-520), and Zmbij on packed pairs."""
import numpy as np

from oracle import cc as O
from ugacc_gb300.generator import make_hamiltonian

ein = lambda s, *a: np.einsum(s, *a, optimize=True)  # noqa: E731


def _amplitudes(no, nv, rng):
    t1, x = 0.1 * rng.standard_normal((no, nv)), 0.1 * rng.standard_normal((no, no, nv, nv))
    return t1, x + x.transpose(1, 0, 3, 2)


def test_two_ring_products():
    no, nv = 3, 5
    H = O.Hamiltonian(make_hamiltonian(no, nv, 2))
    t1, t2 = _amplitudes(no, nv, np.random.default_rng(1))
    V, L = H.V, H.L
    X = 0.5 * t2 + ein("jf,nb->jnfb", t1, t1)
    Wovov = -V("ovov") - ein("jf,mbfe->mbje", t1, V("ovvv")) + ein("nb,mnje->mbje", t1, V("ooov"))
    Wovov = Wovov + ein("mnfe,jnfb->mbje", V("oovv"), X)
    Wovvo = V("ovvo") + ein("jf,mbef->mbej", t1, V("ovvv")) - ein("nb,mnej->mbej", t1, V("oovo"))
    Wovvo = Wovvo - ein("mnef,jnfb->mbej", V("oovv"), X) + 0.5 * ein("mnef,njfb->mbej", L("oovv"), t2)
    t2x = 2 * t2 - t2.transpose(0, 1, 3, 2)
    ref = ein("imae,mbej->ijab", t2x, Wovvo) + ein("imae,mbje->ijab", t2, Wovov) + ein("mjae,mbie->ijab", t2, Wovov)
    ref = ref + ref.transpose(1, 0, 3, 2)

    P = t2.transpose(1, 0, 2, 3) - X
    B = L("ovvo") + ein("jf,mbef->mbej", t1, L("ovvv")) - ein("nb,mnej->mbej", t1, L("oovo"))
    B = B + ein("mnef,jnfb->mbej", L("oovv"), P)
    H_ = ein("imea,mbje->ijab", t2, Wovov)
    half = ein("imae,mbej->ijab", 0.5 * t2x, B) + 0.5 * H_ + H_.transpose(0, 1, 3, 2)
    assert np.abs(half + half.transpose(1, 0, 3, 2) - ref).max() < 1e-14 * 100


def test_zmbij_on_pairs():
    no, nv = 3, 5
    H = O.Hamiltonian(make_hamiltonian(no, nv, 4))
    t1, t2 = _amplitudes(no, nv, np.random.default_rng(2))
    tau = t2 + ein("ia,jb->ijab", t1, t1)
    V = H.V("ovvv")
    e, f = np.triu_indices(nv)
    es, fs = np.triu_indices(nv, 1)
    Vp = V[:, :, e, f] + V[:, :, f, e] * (e != f)
    Vm = V[:, :, es, fs] - V[:, :, fs, es]
    Tp = 0.5 * (tau[:, :, e, f] + tau[:, :, f, e])
    Tm = 0.5 * (tau[:, :, es, fs] - tau[:, :, fs, es])
    S, A = ein("mbp,ijp->mbij", Vp, Tp), ein("mbp,ijp->mbij", Vm, Tm)
    # only i <= j is computed: S is symmetric and A antisymmetric in i <-> j
    assert np.abs(S - S.transpose(0, 1, 3, 2)).max() < 1e-14 and np.abs(A + A.transpose(0, 1, 3, 2)).max() < 1e-14
    assert np.abs(S + A - ein("mbef,ijef->mbij", V, tau)).max() < 1e-14
