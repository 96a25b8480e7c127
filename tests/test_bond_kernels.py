"""The kernels that a size, a width or the number of elements chooses (csrc/bond_fwd.cu, bond_bwd.cu: two channels per lane for
even widths, the general kernels otherwise; csrc/mv_tc.cu: atoms grouped by element; csrc/nlist.cu: a warp or a thread per atom)
at the edges of their ranges, against the numpy fp64 oracle or against one another.

Tolerance of the forces: 1e-5 in the 2-norm.  A force is a sum of about 100 bonds of fp32 terms (6e-8 each) behind a network
of some ten fp32 sums over up to 90 inputs; two orders of summation differ by a few 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm(np.asarray(a) - np.asarray(b)) / np.linalg.norm(b)


def _structures(n_species):
    from grace_runtime_b200 import structures
    rng = np.random.default_rng(5)
    # 110 neighbours inside 6 A: more than one round of staged bonds; and a pair, a triple and a lone atom in an open box
    types, pos, cell, pbc = structures.crystal("fcc", 3.2, (2, 2, 2), n_species=n_species, sigma=0.1, seed=7)
    yield types, pos, cell, pbc
    p = np.array([[5.0, 5, 5], [7.2, 5.5, 5], [20, 20, 20], [22.1, 20, 20.4], [21, 22, 20], [35, 5, 30]])
    yield rng.integers(1, n_species + 1, size=6).astype(np.int32), p, np.eye(3) * 45.0, np.zeros(3, dtype=np.uint8)


@pytest.mark.parametrize("layers,lmax,c1,cr", [
    (1, 4, 32, 0), (1, 4, 8, 0), (1, 4, 34, 0), (1, 3, 64, 0), (1, 3, 18, 0), (1, 2, 16, 0), (1, 2, 6, 0),    # channel pairs
    (1, 4, 9, 0), (1, 3, 33, 0),                                                                             # odd: general kernels
    (2, 3, 32, 16), (2, 3, 20, 6), (2, 2, 32, 16), (2, 2, 8, 10),                                            # four messages, pairs
    (2, 3, 32, 7), (2, 2, 32, 18)])                                                                          # general message kernels
def test_bond_sums_at_the_edges_of_their_widths(backend, tmp_path, layers, lmax, c1, cr):
    from grace_runtime_b200 import modelgen
    from oracle.grace_oracle import GraceOracle
    els = ["Al", "Cu", "Ni"]
    kw = dict(cr=cr, c2=32) if layers == 2 else {}
    path = modelgen.write_model(str(tmp_path / "m.npz"), layers=layers, lmax=lmax, max_order=3, elements=tuple(els), c1=c1, seed=3, **kw)
    system, oracle = backend.System(backend.Model(path), els), GraceOracle(path)
    for types, pos, cell, pbc in _structures(3):
        r = system.compute(types, pos, cell, pbc, energies=True)
        o = oracle.compute(els, types, pos, cell, pbc)
        assert np.abs(r["energies"] - o["energies"]).max() < 1e-5
        assert _rel(r["forces"], o["forces"]) < 1e-5
        assert _rel(r["virial"], o["virial"]) < 1e-5


@pytest.mark.parametrize("cfg,reps,kinds", [("2l", (3, 6, 6), 1), ("2l", (4, 4, 9), 89), ("1l", (3, 3, 22), 40), ("2l", (12, 13, 15), 89)])
def test_atoms_grouped_by_element(backend, tmp_path, monkeypatch, cfg, reps, kinds):
    """one element and many (tiles that hold a few atoms each), the one-block order of the atoms and the one for more than
    8,192 atoms, against the kernels that read every atom's weights by themselves"""
    from grace_runtime_b200 import modelgen, structures
    els = list(modelgen.ELEMENTS)[:kinds]
    path = modelgen.write_config_model(str(tmp_path / "m.npz"), cfg, els, seed=4)
    types, pos, cell, pbc = structures.crystal("fcc", 3.6, reps, n_species=kinds, sigma=0.08, seed=5)
    out = {}
    for mode in ("tc", "ops"):
        monkeypatch.setenv("GRACE_B200_DENSE", mode)
        out[mode] = backend.System(backend.Model(path), els).compute(types, pos, cell, pbc, energies=True)
    assert np.abs(out["tc"]["energies"] - out["ops"]["energies"]).max() < 1e-5
    assert _rel(out["tc"]["forces"], out["ops"]["forces"]) < 1e-5
    assert _rel(out["tc"]["virial"], out["ops"]["virial"]) < 1e-5


@pytest.mark.parametrize("reps", [(4, 4, 5), (6, 6, 8)])
def test_grouped_sums_are_as_exact_as_fp32(backend, tmp_path, monkeypatch, reps):
    """The reduces of a model of order 4 add up to 89 products per row.  fp32 sums are at 2.2e-7 of the fp64 oracle (2-norm of the
    per-atom energies), tensor-core sums that cut off in one accumulator for six products at 1.8e-6: the line is between."""
    from grace_runtime_b200 import modelgen, structures
    from oracle.grace_oracle import GraceOracle
    els = ["Al", "Cu", "Ni", "W"]
    path = modelgen.write_model(str(tmp_path / "m.npz"), elements=tuple(els), seed=0,
                                **dict(modelgen.CONFIGS["1l"], max_order=4, energy_hidden=(64,)))
    types, pos, cell, pbc = structures.crystal("bcc", 3.2, reps, n_species=4, sigma=0.05, seed=9)
    monkeypatch.setenv("GRACE_B200_DENSE", "tc")
    r = backend.System(backend.Model(path), els).compute(types, pos, cell, pbc, energies=True)
    o = GraceOracle(path, spline_n=1024).compute(els, types, pos, cell, pbc)
    assert _rel(r["energies"], o["energies"]) < 6e-7


def test_neighbor_search_on_both_sides_of_its_line(backend, tmp_path):
    """128,000 atoms (a warp per atom) and 160,000 (a thread per atom): copies of one cell have its forces"""
    from grace_runtime_b200 import modelgen, structures
    els = ["Mo", "W"]
    path = modelgen.write_config_model(str(tmp_path / "m.npz"), "1l", els, seed=6)
    types, pos, cell, pbc = structures.crystal("bcc", 3.2, (10, 10, 10), n_species=2, sigma=0.05, seed=8)
    model = backend.Model(path)
    one = backend.System(model, els).compute(types, pos, cell, pbc)
    for reps in ((4, 4, 4), (4, 4, 5)):
        shift = np.stack(np.meshgrid(*[np.arange(k) for k in reps], indexing="ij"), -1).reshape(-1, 3) @ cell
        p = (pos[None] + shift[:, None]).reshape(-1, 3)
        r = backend.System(model, els).compute(np.tile(types, len(shift)), p, cell * np.array(reps)[:, None], pbc)
        assert abs(r["energy"] / len(shift) - one["energy"]) / len(types) < 1e-6
        assert _rel(r["forces"], np.tile(one["forces"], (len(shift), 1))) < 1e-5


def test_groupings_stand_for_sets_of_atoms(backend, tmp_path):
    """Domain-decomposed Systems of a model take turns.  Their element arrays live in buffers of the model that grow and move: when
    the array of one set of a System's atoms comes to lie where the other set's was, its groupings by element must not be taken
    for each other.  Blocks return through the pool of freed device memory; the sizes below make the move happen (a block is taken
    by the first request that is not larger)."""
    from grace_runtime_b200 import modelgen, structures
    els = ["Al", "Cu", "Ni"]
    path = modelgen.write_config_model(str(tmp_path / "m.npz"), "2l", els, seed=4)
    c = structures.crystal("fcc", 3.6, (10, 10, 10), n_species=3, sigma=0.08, seed=5)

    def system(model, n0, n1):
        s = backend.System(model, els, chunksize=600)
        s.set_owned(n0, n1)
        return s

    def energies(s):
        return s.compute(*c, energy_only=True, energies=True)["energies"]
    want = {sizes: energies(system(backend.Model(path), *sizes)) for sizes in ((650, 1400), (1200, 2500))}
    model = backend.Model(path)
    b = system(model, 610, 700)
    energies(b)
    spare = [system(model, 610, 700) for _ in range(6)]    # small blocks for the small requests below
    for s in spare:
        energies(s)
    a = system(model, 650, 1400)
    assert np.abs(energies(a) - want[650, 1400]).max() < 1e-6
    e = system(model, 610, 1250)
    energies(e)
    del s, spare, e             # small blocks, and one for the list of owned atoms that b gets below
    b.set_owned(650, 2500)      # the inner atoms' array grows: the block of a's inner atoms becomes free
    energies(b)
    b.set_owned(1200, 2500)     # the owned atoms' array grows, into that block
    assert np.abs(energies(b) - want[1200, 2500]).max() < 1e-6
    assert np.abs(energies(a) - want[650, 1400]).max() < 1e-6


def test_freed_blocks_count_as_free_memory(backend, tmp_path):
    """Work buffers that a Batch has given back stay in the library's pool.  The automatic pass size of a later call is the one that
    it gets after the pool was returned to the driver (3 %: what else the first call left on the GPU)."""
    import torch
    from grace_runtime_b200 import modelgen, structures
    path = modelgen.write_config_model(str(tmp_path / "m.npz"), "1l", ["W"], seed=6)
    model = backend.Model(path)
    big = structures.crystal("bcc", 3.2, (50, 50, 48), seed=1)
    backend.System(model, ["W"]).release_buffers()
    torch.cuda.empty_cache()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (10 << 30), dtype=torch.uint8, device="cuda")
    try:
        for reps in ((10, 10, 100), (10, 10, 130), (10, 10, 155)):
            types, pos, cell, pbc = structures.crystal("bcc", 3.2, reps, seed=1)
            backend.Batch(model, ["W"]).compute(np.array([len(types)], dtype=np.int32), types, pos, cell[None], pbc[None], energy_only=True)
        before = torch.cuda.mem_get_info()[0]
        chunks = []
        for _ in range(2):
            system = backend.System(model, ["W"])
            system.compute(*big, energy_only=True)
            chunks.append(system.chunksize)
            system.release_buffers()
            del system
        assert before < 9 << 30      # the pool held more than a GB
        assert 0 < chunks[1] < len(big[0]) and abs(chunks[0] - chunks[1]) < 0.03 * chunks[1], chunks
    finally:
        del fill
        torch.cuda.empty_cache()


def _fp64(kind, path, els, c, uq):
    if kind == "3l":
        from oracle.grace3l_oracle import Grace3LOracle
        return Grace3LOracle(path).compute(els, *c)
    from oracle.grace_oracle import GraceOracle
    return GraceOracle(path, spline_n=1024).compute(els, *c, uq=uq)


@pytest.mark.parametrize("kind,reps,copies", [("1l", (6, 7, 7), None), ("2l", (5, 5, 6), None), ("3l", (3, 3, 3), None), ("uq", (5, 5, 6), None),
                                              ("2l", (3, 3, 4), (5, 6, 5)), ("odd", (3, 3, 4), (5, 6, 5))])
def test_tensor_core_sums_are_no_further_off_than_fp32(backend, tmp_path, monkeypatch, kind, reps, copies):
    """Errors against the fp64 oracle of the tensor-core operations and of the fp32 kernels (GRACE_B200_DENSE=ops), root mean square of
    two structures: at few atoms, where the small products have accumulators of their own, and above 18,944 atoms (copies of a
    cell), where the usual widths go without and others (odd: 24, 12 and 40 channels) do not.  The margins: the two errors are
    of 2 x 50 atoms at least and hardly correlated, they scatter by 20 % (energies, forces); the grade's, of fewer and smaller sums, by
    twice that.  With two tf32 parts per operand the ratios were 1.6 (GRACE-3L) and 16 (grade)."""
    from grace_runtime_b200 import modelgen, modelgen3l, structures
    els = ["Al", "Cu", "Ni", "W"]
    path, lattice, a = str(tmp_path / "m.npz"), "fcc", 3.6
    if kind == "3l":
        lattice, a = "bcc", 3.2
        modelgen3l.write_model_3l(path, elements=els, lmax=4, channels=(64, 64, 64), rho_width=32, embedding=16, radial_hidden=128,
                                  energy_hidden=64, rcut=6.0, avg_neigh=58.0, seed=0)
    elif kind == "uq":
        plain = modelgen.write_model(path + ".plain.npz", elements=tuple(els), seed=0, **dict(modelgen.CONFIGS["2l"], max_order=4, lmax=2))
        modelgen.add_uq_head(plain, path, seed=0)
    elif kind == "odd":
        modelgen.write_model(path, elements=tuple(els), seed=0, **dict(modelgen.CONFIGS["2l"], c1=24, cr=12, c2=40))
    else:
        lattice, a = ("bcc", 3.2) if kind == "1l" else (lattice, a)
        modelgen.write_config_model(path, kind, els, seed=0)
    err = {}
    for seed in (1, 2):
        types, pos, cell, pbc = structures.crystal(lattice, a, reps, n_species=4, sigma=0.06, seed=seed)
        o = _fp64(kind, path, els, (types, pos, cell, pbc), kind == "uq")
        m = 1
        if copies:
            shift = np.stack(np.meshgrid(*[np.arange(k) for k in copies], indexing="ij"), -1).reshape(-1, 3) @ cell
            m, pos = len(shift), (pos[None] + shift[:, None]).reshape(-1, 3)
            types, cell = np.tile(types, m), cell * np.array(copies)[:, None]
        for mode in ("tc", "ops"):
            monkeypatch.setenv("GRACE_B200_DENSE", mode)
            r = backend.System(backend.Model(path), els).compute(types, pos, cell, pbc, energies=True, uq=kind == "uq")
            for q in ("energies", "forces", "gamma"):
                if q in o and q in r:
                    err.setdefault((q, mode), []).append(_rel(r[q], np.tile(o[q], (m,) + (1,) * (o[q].ndim - 1))))
    for q, mode in err:
        if mode == "tc":
            e = {k: np.sqrt(np.mean(np.square(err[q, k]))) for k in ("tc", "ops")}
            assert e["tc"] < (1.4 if q == "gamma" else 1.2) * e["ops"], (q, e)


@pytest.mark.parametrize("layers,lmax", [(1, 2), (1, 3), (1, 4), (2, 2), (2, 3)])
@pytest.mark.parametrize("neighbours", [64, 66, 97, 98, 124, 125, 129])
def test_bond_sums_at_the_edges_of_their_rounds(backend, tmp_path, layers, lmax, neighbours):
    """A cluster in which every atom sees all the others: as many bonds as a round of the reverse kernels holds, and one more (csrc/
    bond_bwd.cu: 65, 97, 124 or the 128 threads; the forward kernels stage 96)."""
    from grace_runtime_b200 import modelgen
    from oracle.grace_oracle import GraceOracle
    els = ["Al", "Cu", "Ni"]
    path = modelgen.write_config_model(str(tmp_path / "m.npz"), "1l" if layers == 1 else "2l", els, seed=3) if lmax == 5 - layers else \
        modelgen.write_model(str(tmp_path / "m.npz"), layers=layers, lmax=lmax, max_order=3, elements=tuple(els), seed=3)
    rng = np.random.default_rng(neighbours)
    g = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij"), -1).reshape(-1, 3) * 0.9
    g = g[np.argsort((g * g).sum(1) + 1e-3 * rng.random(len(g)))][:neighbours + 1] + 0.1 * (rng.random((neighbours + 1, 3)) - 0.5)
    assert np.linalg.norm(g[:, None] - g[None], axis=2).max() < 6.0
    types = rng.integers(1, 4, size=len(g)).astype(np.int32)
    args = (types, g + 20.0, np.eye(3) * 40.0, np.zeros(3, dtype=np.uint8))
    r, o = backend.System(backend.Model(path), els).compute(*args, energies=True), GraceOracle(path, spline_n=1024).compute(els, *args)
    assert _rel(r["energies"], o["energies"]) < 1e-5
    assert _rel(r["forces"], o["forces"]) < 1e-5
    assert _rel(r["virial"], o["virial"]) < 1e-5


@pytest.mark.parametrize("cr", [16, 6, 7])
def test_message_gradients_by_atomics(backend, tmp_path, monkeypatch, cr):
    """GRACE_B200_MSG_ATOMICS: what a call does whose buffer of message-gradient shares cannot be had - the reverse message kernels
    (two channels per lane for 16 and 6, one for 7) add the shares of dE/dmsg atomically: the same forces."""
    from grace_runtime_b200 import modelgen, structures
    els = ["Al", "Cu", "Ni"]
    path = modelgen.write_model(str(tmp_path / "m.npz"), layers=2, lmax=3, max_order=3, elements=tuple(els), cr=cr, c2=32, seed=3)
    c = structures.crystal("fcc", 3.4, (3, 3, 2), n_species=3, sigma=0.1, seed=7)
    model = backend.Model(path)
    a = backend.System(model, els).compute(*c)
    monkeypatch.setenv("GRACE_B200_MSG_ATOMICS", "1")
    b = backend.System(model, els).compute(*c)
    assert _rel(b["forces"], a["forces"]) < 1e-5
    assert _rel(b["virial"], a["virial"]) < 1e-5
