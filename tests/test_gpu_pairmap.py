"""The pair-factorised single-vector map (csrc/pairmap.cu) against the oracle's product and the
candidate map, over the forms it accepts and at the edges of its tables: class sizes below, at and
above the instantiated ones up to 32 pairs, orbital 63, rows with different particle numbers, bases
that miss targets, non-Hermitian lists, H(u) = A + u B at several u, amplitudes set anew; operators
it refuses go to the hit records.

Bars: complex128 within 1e-13 relative of the oracle, complex64 within 2e-6 (another order of the
same products, as for the other maps).
"""
import os
from contextlib import contextmanager

import numpy as np
import pytest

import oracle as O
import momed

pytestmark = pytest.mark.gpu


@contextmanager
def env(**kv):
    old = {k: os.environ.get(k) for k in kv}
    os.environ.update({k: str(v) for k, v in kv.items()})
    try:
        yield
    finally:
        for k, v in old.items():
            if v is None:
                del os.environ[k]
            else:
                os.environ[k] = v


@pytest.fixture(scope="module")
def h():
    with env(MOMED_PAIRMAP=1):             # whatever the size: these sectors are far below the size rule
        hd = momed.Handle(0)
        yield hd
        hd.close()


def rel(a, b):
    return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))


def pair_terms(a, b, ncc, seed, hermitian=True, keep=1.0):
    """All momentum-conserving two-body terms on an a x b mesh of ncc components plus a one-body
    diagonal: (amp, in, out) sorted by (in, out)."""
    nk = a * b
    orb = np.arange(nk * ncc)
    x, y, c = orb % nk % a, orb % nk // a, orb // nk
    p, q = np.triu_indices(len(orb), 1)
    key = ((x[p] + x[q]) % a * b + (y[p] + y[q]) % b) * 4 + c[p] + c[q]
    masks = (np.uint64(1) << p.astype(np.uint64)) | (np.uint64(1) << q.astype(np.uint64))
    rng = np.random.default_rng(seed)
    o, i = np.nonzero(key[:, None] == key[None, :])
    m = rng.standard_normal((len(p), len(p))) + 1j * rng.standard_normal((len(p), len(p)))
    take = rng.random(m.shape) < keep
    if hermitian:
        m = (m + m.conj().T) / 2
        take = np.triu(take) | np.triu(take).T
    sel = take[o, i]
    o, i = o[sel], i[sel]
    one = np.uint64(1) << orb.astype(np.uint64)
    amp = np.concatenate([m[o, i], rng.standard_normal(len(orb)) + 0j])
    out, in_ = np.concatenate([masks[o], one]), np.concatenate([masks[i], one])
    order = np.lexsort((out, in_))
    return amp[order], in_[order], out[order]


def full_list(amp, in_, out):
    f = np.zeros(len(amp), O.SCAT_DTYPE)
    f["re"], f["im"], f["out"], f["in"] = amp.real, amp.imag, out, in_
    f["pm"] = [momed.parity_mask(int(o)) ^ momed.parity_mask(int(i)) for o, i in zip(out, in_)]
    return f


def vec(n, seed=3):
    rng = np.random.default_rng(seed)
    return rng.standard_normal(n) + 1j * rng.standard_normal(n)


def check(h, basis, amp, in_, out):
    h.set_basis(basis)
    h.set_scatter(amp, in_, out)
    x = vec(len(basis))
    ref = O.matvec(basis, full_list(amp, in_, out), x)
    with env(MOMED_HITCACHE=0):
        cand = h.matvec(x)
    info = h.build_hit_cache()
    assert rel(h.matvec(x), ref) < 1e-13 and rel(cand, ref) < 1e-13
    assert rel(h.matvec(x.astype(np.complex64)).astype(np.complex128), ref) < 2e-6
    assert info["hits"] == h.build_sparse() - len(basis)      # the off-diagonal hits, counted another way
    h.release_sparse()


def sector(a, b, ne, i):
    subs, _ = O.momentum_subspaces(O.mesh_klist(a, b), (a, b), ne, Nc_conserve=len(ne))
    return subs[i]


# classes of 5-6, 7, 7-8, 10, 12, 13-14 and 14-15 pairs; two components: 5-6 and 12, 7 and 15, 11-12 and 24
@pytest.mark.parametrize("a,b,ne,i", [(3, 4, (2,), 1), (3, 4, (5,), 0), (3, 5, (5,), 4), (4, 4, (6,), 3), (3, 7, (5,), 2),
                                      (5, 5, (4,), 7), (4, 7, (4,), 1), (3, 10, (4,), 29), (4, 3, (2, 3), 5),
                                      (3, 5, (3, 2), 2), (4, 6, (2, 2), 11), (4, 6, (0, 3), 1)])
def test_map_matches_oracle(h, a, b, ne, i):
    check(h, sector(a, b, ne, i), *pair_terms(a, b, len(ne), 1))


def test_classes_of_32_pairs_and_orbital_63(h):
    subs, _ = O.momentum_subspaces(O.mesh_klist(4, 8), (4, 8), (2, 1), Nc_conserve=2)
    basis = subs[9]
    assert int(basis[-1]) >> 63 == 1
    check(h, basis, *pair_terms(4, 8, 2, 2))


def test_non_hermitian_list_and_missing_couplings(h):
    check(h, sector(3, 6, (5,), 2), *pair_terms(3, 6, 1, 3, hermitian=False))
    check(h, sector(3, 6, (5,), 2), *pair_terms(3, 6, 1, 4, keep=0.6))


def test_basis_that_misses_targets_and_mixes_particle_numbers(h):
    rng = np.random.default_rng(6)
    t = pair_terms(3, 5, 1, 5)
    some = sector(3, 5, (5,), 1)
    check(h, some[rng.random(len(some)) < 0.6], *t)
    mixed = np.unique(np.concatenate([sector(3, 5, (n,), s) for n, s in ((1, 0), (3, 2), (4, 3), (6, 1))]))
    check(h, mixed, *t)
    check(h, np.array([0b11, 0b101, 1 << 14], np.uint64), *t)
    check(h, np.array([0b1], np.uint64), *t)                 # no pairs at all: refused, the records serve


def test_parametrised_operator_follows_u_and_new_amplitudes(h):
    amp, in_, out = pair_terms(3, 6, 1, 7)
    basis = sector(3, 6, (6,), 4)
    rng = np.random.default_rng(8)
    amp_b = amp * rng.choice([0.0, 1.0, 0.5], len(amp))
    herm = amp_b.copy()
    pos = {(int(i), int(o)): k for k, (i, o) in enumerate(zip(in_, out))}
    for k, (i, o) in enumerate(zip(in_, out)):
        herm[pos[(int(o), int(i))]] = np.conj(herm[k])
    x = vec(len(basis))
    for scale in (1.0, -2.0):
        h.set_basis(basis)
        h.set_scatter_pair(scale * amp, herm, in_, out)
        h.build_hit_cache()
        for u in (1.0, 0.0, 1.7):
            h.set_param(u)
            ref = O.matvec(basis, full_list(scale * amp + u * herm, in_, out), x)
            assert rel(h.matvec(x), ref) < 1e-13
            assert rel(h.matvec(x.astype(np.complex64)).astype(np.complex128), ref) < 2e-6
            w = np.linalg.eigvalsh(O.dense_hamiltonian(basis, full_list(scale * amp + u * herm, in_, out)))[:3]
            for prec in (0, 1):                              # FP64 and mixed solves over the same tables
                v, _, _, _ = h.eigsolve(3, tol=1e-12, precision=prec, want_vectors=False)
                assert np.max(np.abs(v - w) / np.abs(w)) < 1e-10
            v, _, _, _ = h.batch_solve([0.3], 3, tol=1e-12)
            w = np.linalg.eigvalsh(O.dense_hamiltonian(basis, full_list(scale * amp + 0.3 * herm, in_, out)))[:3]
            assert np.max(np.abs(v[0] - w) / np.abs(w)) < 1e-10
    h.set_param(1.0)


def test_operators_without_the_pair_form(h):
    basis = sector(3, 5, (5,), 1)
    amp, in_, out = pair_terms(3, 5, 1, 9)
    few = (in_ == out) | ((in_ ^ out) % np.uint64(7) == 0)
    check(h, basis, amp[few], in_[few], out[few])            # few couplings per pair
    twice = np.concatenate([np.arange(len(amp)), [40, 41]])
    check(h, basis, amp[twice], in_[twice], out[twice])      # terms listed twice
    hop = np.array([1.0 + 0.5j, 1.0 - 0.5j])                 # a one-body term off the diagonal
    check(h, np.arange(1, 256, dtype=np.uint64), np.concatenate([amp, hop]),
          np.concatenate([in_, np.array([1, 2], np.uint64)]), np.concatenate([out, np.array([2, 1], np.uint64)]))
    p, q = np.triu_indices(9, 1)                             # no conservation: one class of 36 pairs
    m = (np.uint64(1) << p.astype(np.uint64)) | (np.uint64(1) << q.astype(np.uint64))
    rng = np.random.default_rng(10)
    v = rng.standard_normal((36, 36))
    check(h, np.array([s for s in range(512) if bin(s).count("1") == 4], np.uint64), (v + v.T).reshape(-1) + 0j,
          np.tile(m, 36), np.repeat(m, 36))


def test_repeated_products_build_the_tables_unreported(h):
    """From the second momed_matvec on a basis and operator the map runs over the pair tables; the
    hit cache stays what the caller asked for."""
    amp, in_, out = pair_terms(3, 6, 1, 11)
    basis = sector(3, 6, (6,), 2)
    h.set_basis(basis)
    h.set_scatter(amp, in_, out)
    ref = lambda x: O.matvec(basis, full_list(amp, in_, out), x)
    for seed in range(4):
        x = vec(len(basis), seed)
        assert rel(h.matvec(x), ref(x)) < 1e-13
        assert h.hit_cache_info() is None
    h.set_basis(basis[::2].copy())
    x = vec(len(basis[::2]))
    for _ in range(3):
        assert rel(h.matvec(x), O.matvec(basis[::2], full_list(amp, in_, out), x)) < 1e-13
    h.set_hbm_budget(1 << 34)                                # a budgeted handle allocates nothing by itself
    h.set_basis(basis)
    for _ in range(3):
        assert rel(h.matvec(vec(len(basis))), ref(vec(len(basis)))) < 1e-13
    h.set_hbm_budget(0)


def test_size_and_density_rules(h):
    """By size and density: a 3x9 sector (6.2M entries, 6 hits each) takes the pair form, a half-filled
    4x6 one (5.7M entries, 3.4 hits each) is declined and runs over the records; same products."""
    with env(MOMED_PAIRMAP=2):
        for a, b, ne, i in ((3, 9, (9,), 5), (4, 6, (11,), 2)):
            check(h, sector(a, b, ne, i), *pair_terms(a, b, 1, 12))
