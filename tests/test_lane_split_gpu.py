"""Quartets shared by several lanes (GPU tests).

Lists with few quartets and long primitive loops are launched with 2^glog
lanes per quartet (Segments in csrc/pfk_device.cuh).  cc-pVDZ has shells of
1, 4 and 9 primitives, so its quartets' loops are 1 to 6561 long and the
segments of one list take 1 to 32 lanes each; 1 x 81 and 81 x 1 pairs put
all lanes on one side.  Against the oracle's tensor within 1e-10, as the
one-lane kernels: the lanes' sums only change the order of the additions."""
import numpy as np
import pytest

import oracle
from helpers import alkane, basis_library, pfk, random_density, regression_cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["ethylene", "methane"])
def molecule(request):
    atoms = regression_cases()["ethylene_rhf_ccpvdz_auto"]["atoms"] if request.param == "ethylene" else alkane(1)
    ob = oracle.Basis(oracle.shells_for(oracle.Molecule(atoms), "cc-pvdz"))
    eri, _ = ob.eri_tensor(1e-10, oracle.OS)
    return pfk().shells_for(atoms, "cc-pvdz", basis_library())[1], eri


@pytest.mark.parametrize("engine", ["os", "rys"])
def test_builds_and_tensor(molecule, engine):
    shells, eri = molecule
    eng = pfk().FockEngine(shells, engine=engine)
    nb = eng.nbasis
    Pa, Pb = random_density(nb, seed=41), random_density(nb, seed=42)
    G = eng.fock_rhf(Pa)
    assert np.abs(G - oracle.fock_rhf_tensor(eri, Pa)).max() < 1e-10
    Ga, Gb = eng.fock_uhf(Pa, Pb)
    Gao, Gbo = oracle.fock_uhf_tensor(eri, Pa, Pb)
    assert max(np.abs(Ga - Gao).max(), np.abs(Gb - Gbo).max()) < 1e-10
    assert np.abs(eng.eri_tensor() - eri).max() < 1e-10
    # shards cut every segment; three of them leave some segments empty
    parts = []
    for n in (2, 3, 7):
        total = np.zeros_like(G)
        for r in range(n):
            eng.set_shard(r, n)
            total += eng.fock_rhf(Pa)
        parts.append(np.abs(total - G).max())
    eng.set_shard(0, 1)
    assert max(parts) < 1e-12
    assert np.array_equal(eng.fock_rhf(Pa), G)
    eng.close()


def test_mixed_and_density_screened(molecule):
    """FP32 lists have segments of their own; a density screen below every
    contribution changes nothing, one above everything leaves nothing."""
    shells, eri = molecule
    eng = pfk().FockEngine(shells, precision="mixed", fp32_bound=1e-6)
    P = random_density(eng.nbasis, seed=43)
    ref = oracle.fock_rhf_tensor(eri, P)
    G = eng.fock_rhf(P)
    # FP32 quartets are below 1e-6 each, relative error a few 2^-24 of them
    assert np.abs(G - ref).max() < 1e-8
    eng.set_density_screening(1e-30)
    assert np.array_equal(eng.fock_rhf(P), G)
    eng.set_density_screening(1e30)
    assert not eng.fock_rhf(P).any()
    eng.close()
