"""Row-driven product against the partitioned pipeline on a GB300: the same terms,
summed exactly in another order, so keys, amplitudes and <v|Hv> are equal bit
for bit.  A context with a device budget always takes the partitioned pipeline."""
import numpy as np
import pytest

import sfci_gb300 as sg
from sfci_gb300 import fcidump as fd

pytestmark = pytest.mark.gpu

# spatial orbitals, integrals, alpha and beta electrons, sources, then lambda, coefficient, capacity, cut, top Nd
CASES = {
    "small strings, every slot hot": (10, "rhf", 5, 5, 9000, 0.0, 1.0, 100000, 1e-5, 0),
    "unequal spins": (12, "rhf", 3, 6, 6000, 1.25, -0.5, 100000, 1e-5, 0),
    "one electron of a spin": (20, "rhf", 1, 6, 9000, 0.0, 1.0, 400000, 1e-6, 0),
    "one hole of a spin": (16, "rhf", 15, 5, 3000, 0.5, 2.0, 100000, 1e-5, 0),
    "oriented alpha-beta integrals": (14, "uhf", 6, 6, 3000, 0.0, 1.0, 400000, 1e-6, 0),
    "32 orbitals of a spin": (32, "rhf", 4, 5, 3001, 0.0, 1.0, 2000000, 1e-7, 0),
    "two-word keys": (34, "rhf", 5, 5, 5003, -1.5, 1.0, 2000000, 1e-7, 0),
    "accumulators for more than 2^15 terms": (34, "rhf", 8, 8, 1201, 0.0, 1.0, 2000000, 1e-6, 0),
    "output capped, top of the input": (20, "rhf", 6, 6, 9000, 2.0, 0.25, 3000, 1e-6, 6001),
    "no cut, output capped below the survivors": (20, "rhf", 5, 5, 6000, 0.0, 1.0, 200000, -1.0, 0),
}


def vector(M, na, nb, n, rng):
    """n distinct determinants near the lowest one, two words each, sorted by key."""
    got = set()
    p = np.exp(-np.arange(M) / (0.35 * M))
    while len(got) < n:
        a = rng.choice(M, na, replace=False, p=p / p.sum())
        for _ in range(24):  # several beta strings to an alpha string
            b = rng.choice(M, nb, replace=False, p=p / p.sum())
            got.add(sum(1 << 2 * int(i) for i in a) | sum(2 << 2 * int(i) for i in b))
            if len(got) == n:
                break
    keys = sg.keys_from_ints(sorted(got), 1 if M <= 32 else 2)
    amps = rng.standard_normal(n) * np.exp(-rng.uniform(0.0, 12.0, n))
    return keys, amps / np.linalg.norm(amps)


@pytest.mark.parametrize("name", list(CASES))
def test_row_form_gives_the_partitioned_product(name, tmp_path):
    M, kind, na, nb, n, lam, coeff, cap, cut, nd = CASES[name]
    path = str(tmp_path / "sys_IN")
    if kind == "rhf":
        fd.rhf_to_in_file(path, M, na + nb, 3)
    else:
        fd.uhf_to_in_file(path, M, na + nb, 2, 3)
    keys, amps = vector(M, na, nb, n, np.random.default_rng(7))
    got = []
    for budget in (0, 64 << 30):
        c = sg.Context(path, 2 * M, na + nb, Nd=nd or n, coeff_cut=cut, mem_budget=budget)
        v, out = c.vec_from(keys, amps), c.vec(cap)
        for _ in range(2):  # the second product is planned from the first one's statistics
            d = c.SpMVMtply_bucket(v, out, lam, coeff)
        got.append((*out.download(), d, c.last_stats()))
    (k, a, d, st), (k0, a0, d0, st0) = got
    assert st["leaves"] != st0["leaves"]  # work units against hash leaves: two routes
    assert np.array_equal(k, k0)
    assert np.array_equal(a.view(np.uint64), a0.view(np.uint64))
    assert d == d0
    assert [st[x] for x in ("terms", "unique")] == [st0[x] for x in ("terms", "unique")]


def test_inputs_the_row_form_declines(tmp_path):
    """Mixed spin counts, a repeated key and terms beyond the row accumulators give
    what they gave: the partitioned pipeline's product, or its range error."""
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, 14, 10, 3)
    rng = np.random.default_rng(11)
    k1, a1 = vector(14, 5, 5, 2500, rng)
    k2, a2 = vector(14, 4, 6, 2500, rng)
    mixed = np.concatenate([k1, k2])
    twice = np.concatenate([k1, k1[:1]])
    for keys, amps, fails in ((mixed, np.concatenate([a1, a2]), False), (twice, np.concatenate([a1, a1[:1]]), False),
                              (k1, a1 * 2.0 ** 17, False), (k1, a1 * 2.0 ** 40, True)):
        got = []
        for budget in (0, 64 << 30):
            c = sg.Context(path, 28, 10, Nd=len(amps), mem_budget=budget)
            v, out = c.vec_from(keys, amps), c.vec(400000)
            if fails:
                with pytest.raises(sg.SfciError) as e:
                    c.SpMVMtply_bucket(v, out, 0.0, 1.0)
                assert e.value.status == "SFCI_ERR_NUMERIC"
                continue
            d = c.SpMVMtply_bucket(v, out, 0.0, 1.0)
            got.append((*out.download(), d))
        if not fails:
            assert np.array_equal(got[0][0], got[1][0]) and got[0][2] == got[1][2]
            assert np.array_equal(got[0][1].view(np.uint64), got[1][1].view(np.uint64))


@pytest.mark.parametrize("M,na,nb,n", [(14, 5, 5, 2500), (28, 5, 6, 1200), (34, 5, 5, 1601)])
def test_extra_sources_join_their_rows(M, na, nb, n, tmp_path):
    """The linear solver's product (two vectors removed before the cut): extra terms
    on determinants the product reaches, and on some far from every source, whose
    rows hold nothing else."""
    path = str(tmp_path / "sys_IN")
    fd.rhf_to_in_file(path, M, na + nb, 3)
    rng = np.random.default_rng(13)
    keys, amps = vector(M, na, nb, n, rng)
    far = sorted({sum(1 << 2 * int(i) for i in M - 1 - np.arange(na)) |
                  sum(2 << 2 * int(i) for i in M - 1 - rng.choice(M // 2, nb, replace=False)) for _ in range(40)})
    far = sg.keys_from_ints(far, 1 if M <= 32 else 2)
    basis = [(np.concatenate([keys[1::3], far]), rng.standard_normal(len(keys[1::3]) + len(far))),
             (keys[::2], rng.standard_normal(len(keys[::2]))), (keys, amps)]
    got = []
    for budget in (0, 64 << 30):
        c = sg.Context(path, 2 * M, na + nb, Nd=n, coeff_cut=1e-7, mem_budget=budget)
        vecs = [c.vec_from(k, a) for k, a in basis]
        out = c.vec(2000000)
        for pair in (vecs, vecs[::2]):
            h = c.spmspvm_bucket_linear(vecs[2], out, 0.75, pair)
            got.append((*out.download(), h, c.last_stats()["terms"]))
    for x, y in zip(got[:2], got[2:]):
        assert np.array_equal(x[0], y[0]) and np.array_equal(x[1].view(np.uint64), y[1].view(np.uint64))
        assert np.array_equal(x[2], y[2]) and x[3] == y[3]
