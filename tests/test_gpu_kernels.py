"""Edge sizes of the solver's kernels (GPU): one block row up to several CTAs'
worth, every block size, isolated nodes (banks without couplings)."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def block_system(nb, bs, seed, isolated=0, reach=40, degree=6):
    """Symmetric, strictly diagonally dominant block system on nb nodes of a
    random graph with couplings up to `reach` nodes apart; the last `isolated`
    nodes couple to nothing (their rows have off-diagonals inside the node)."""
    rng = np.random.default_rng(seed)
    m = max(nb - isolated, 1)
    i = rng.integers(0, m, size=degree * m // 2)
    j = np.clip(i + rng.integers(1, reach + 1, size=len(i)), 0, m - 1)
    keep = i != j
    G = sp.csr_matrix((np.ones(int(keep.sum())), (i[keep], j[keep])), shape=(nb, nb))
    G = ((G + G.T) != 0).astype(np.float64) + sp.identity(nb)
    B = sp.kron(G, np.ones((bs, bs)), format="csr")
    B.data = rng.uniform(-1.0, 1.0, size=B.nnz)
    A = (B + B.T) * 0.5
    A = A - sp.diags(A.diagonal())
    d = np.asarray(abs(A).sum(axis=1)).ravel() + rng.uniform(0.5, 1.5, size=nb * bs)
    A = (A + sp.diags(d)).tocsc()
    A.sum_duplicates()
    A.sort_indices()
    return A


def make_solver(bs, precision="fp64", extra=None, **params):
    import lss
    gb = {"precision": precision}
    gb.update(extra or {})
    return lss.Solver.create({"solver": "GPUHybrid", "GPUHybrid": {"block_size": bs, **params}, "gb300": gb})


@pytest.mark.parametrize("bs", [1, 2, 3])
@pytest.mark.parametrize("nb,isolated", [(1, 0), (2, 1), (31, 0), (33, 0), (70, 64), (129, 0), (1100, 200), (5000, 1500)])
def test_mas_apply_edge_sizes(bs, nb, isolated, built):
    """MAS against the CPU restatement on the same partition.  The blocks are
    diagonally dominant with a condition number of at most a few hundred, so the two
    FP64 inverses differ by less than 1e-12 relative and the FP32 ones by
    less than 1e-4; coarse vectors and uncoupled banks add exact copies."""
    from oracle import oracle as O
    A = block_system(nb, bs, seed=nb + bs, isolated=isolated)
    params = {"block_size": bs, "do_hybrid_precond": False}
    r = np.random.default_rng(nb).standard_normal(A.shape[0])
    zo = None
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-4)):
        s = make_solver(bs, precision, do_hybrid_precond=False)
        s.factorize(A)
        if zo is None:
            perm, offs = s.partition()
            zo = O.CpuSolver(A, params, perm=perm, part_offsets=offs).precond(r)
        z = s.mas_apply(r)
        assert np.linalg.norm(z - zo) <= tol * np.linalg.norm(zo), (precision, nb)
        np.testing.assert_array_equal(s.mas_apply(r), z)  # fixed order of every sum
        s.close()


@pytest.mark.parametrize("bs", [1, 2, 3])
@pytest.mark.parametrize("m", [1, 24, 25, 49, 97, 160, 161, 384, 390, 900, 1700])
def test_stiff_apply_edge_sizes(bs, m, built):
    """A_SS^-1 r on m given DOFs: every warp split of the dense apply, its
    limit (160), one multifrontal front, a tree, fronts of several row chunks.
    Diagonally dominant blocks (condition at most a few hundred): 1e-12 of a
    dense solve."""
    nb = 2400 // bs
    A = block_system(nb, bs, seed=7 * m + bs)
    dofs = np.arange(5, 5 + m)
    s = make_solver(bs, extra={"composition": "additive"}, select_bad_dofs_from_l1_norm=False,
                    decompose_subdomains=False, expand_subdomains=False)
    s.set_problematic_dofs(dofs)
    s.factorize(A)
    np.testing.assert_array_equal(s.selected_dofs(), dofs)
    r = np.random.default_rng(m).standard_normal(A.shape[0])
    d = s.precond(r) - s.mas_apply(r)
    x = np.linalg.solve(A.T[dofs][:, dofs].toarray(), r[dofs])
    scale = np.linalg.norm(s.mas_apply(r)[dofs])  # the difference cancels the MAS part
    assert np.linalg.norm(d[dofs] - x) <= 1e-12 * (np.linalg.norm(x) + scale)
    rest = np.ones(A.shape[0], bool)
    rest[dofs] = False
    assert np.all(d[rest] == 0.0)
    s.close()


@pytest.mark.parametrize("m", [8001, 16002, 30000])
def test_stiff_apply_long_row_chunks(m, built):
    """A_SS^-1 r where a level of the tree has more CTAs than the GPU holds at 64
    rows each (1.4k, 2.8k and 5.3k): chunks of 128 to 512 rows, with
    remainders.  Diagonally dominant as above: 1e-12 of a sparse LU."""
    import scipy.sparse.linalg as spla
    A = block_system(11000, 3, seed=m)
    dofs = np.arange(5, 5 + m)
    s = make_solver(3, extra={"composition": "additive"}, select_bad_dofs_from_l1_norm=False,
                    decompose_subdomains=False, expand_subdomains=False)
    s.set_problematic_dofs(dofs)
    s.factorize(A)
    r = np.random.default_rng(m).standard_normal(A.shape[0])
    z = s.mas_apply(r)
    d = s.precond(r) - z
    np.testing.assert_array_equal(s.precond(r) - z, d)  # fixed order of every sum
    s.close()
    x = spla.splu(A[dofs][:, dofs].tocsc()).solve(r[dofs], trans="T")
    assert np.linalg.norm(d[dofs] - x) <= 1e-12 * (np.linalg.norm(x) + np.linalg.norm(z[dofs]))


@pytest.mark.parametrize("nodes", [100, 300, 2000])
def test_info_reports_the_tree_of_fronts(nodes, built):
    """get_info's multifrontal counts are those of the host plan: one front, a
    joined front, a tree with splits in two.  The subdomain is a chain of nodes,
    whose tree has the same levels and fronts in the solver's order."""
    import lss
    chain = sp.diags([1.0, 4.0, 1.0], [-1, 0, 1], shape=(2100, 2100))
    A = sp.kron(chain, np.ones((3, 3)) + sp.identity(3), format="csc")
    A.sort_indices()
    dofs = np.arange(30, 30 + 3 * nodes)
    s = make_solver(3, select_bad_dofs_from_l1_norm=False, decompose_subdomains=False, expand_subdomains=False)
    s.set_problematic_dofs(dofs)
    s.factorize(A)
    info, plan = s.get_info(), lss.stiff_elimination_tree(A, 3, dofs)
    s.close()
    assert (info["multifrontal_levels"], info["multifrontal_fronts"]) == (plan["levels"], plan["fronts"])


@pytest.mark.parametrize("n", [3, 96, 3000])
def test_double_float_split_matches_casts(n, built):
    """The FP64 <-> FP32 conversions on the integer pipe equal the casts bit for
    bit: through A = I the double-float product returns fl32(x) + fl32(x -
    fl32(x)) exactly, for every sign, zeros, ties, denormal and extreme exponents."""
    s = make_solver(3, "mixed", do_hybrid_precond=False)
    s.factorize(sp.identity(n, format="csc"))
    rng = np.random.default_rng(n)
    for scale in (0, 30, 60, 126, 160):
        x = rng.standard_normal(n) * 2.0 ** rng.uniform(-scale, min(scale, 100), size=n)
        x[::7] = 0.0
        x[1::11] = np.float64(np.float32(x[1::11])) * (1.0 + 2.0 ** -24)  # a tie of the high word
        x[2::13] = np.float32(x[2::13])                                    # no low word
        hi = x.astype(np.float32)
        lo = (x - hi.astype(np.float64)).astype(np.float32)
        np.testing.assert_array_equal(s.spmv_outer(x), hi.astype(np.float64) + lo.astype(np.float64))
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("hybrid", [True, False])
def test_refactorized_solves_match_fresh_ones(precision, hybrid, built):
    """The iterations captured for one factorization serve later ones of the
    pattern: solves after a change of values, of the stiff set (other sizes,
    none) and back equal those of a new solver bit for bit."""
    from lss import gen
    rng = np.random.default_rng(4)
    n = (11, 10, 9)
    E, _ = gen.sphere_inclusion_E(*n, np.random.Generator(np.random.PCG64(5)), radius=0.2, E_in=1e4)
    F, _ = gen.sphere_inclusion_E(*n, np.random.Generator(np.random.PCG64(6)), radius=0.3, E_in=1e5)
    mats = [gen.elasticity_cube(*n, e) for e in (E, F, np.ones_like(E), 1.7 * E, E)]
    b = rng.standard_normal(mats[0].shape[0])
    params = {"gmm_jump_threshold": 10.0, "min_subdomain_size": 4, "do_hybrid_precond": hybrid}
    kept = make_solver(3, precision, **params)
    first = None
    for k, A in enumerate(mats):
        kept.factorize(A)
        x = kept.solve(b)
        fresh = make_solver(3, precision, **params)
        fresh.factorize(A)
        np.testing.assert_array_equal(x, fresh.solve(b), err_msg=str(k))
        np.testing.assert_array_equal(kept.solve(b), x)
        if first is None:
            first = x
        fresh.close()
    np.testing.assert_array_equal(x, first)
    kept.close()


@pytest.mark.parametrize("max_iter", [0, 1, 3, 4, 5, 9])
def test_iteration_limit(max_iter, built):
    """The limit holds whatever its place in a chunk of iterations, and a solve
    from the point it left continues to convergence."""
    A = block_system(700, 3, seed=1)
    b = np.random.default_rng(2).standard_normal(A.shape[0])
    s = make_solver(3, do_hybrid_precond=False, max_iter=max_iter)
    s.factorize(A)
    x = s.solve(b)
    info = s.get_info()
    assert info["num_iterations"] == max_iter and info["status"] == "max_iterations"
    s.set_parameters({"GPUHybrid": {"max_iter": 1000}})
    y = s.solve(b, x.copy())
    assert s.get_info()["status"] == "converged_rel"
    assert np.linalg.norm(b - A.T @ y) <= 1e-10 * np.linalg.norm(b)
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bs", [1, 2, 3])
@pytest.mark.parametrize("nb,isolated", [(1, 0), (2, 1), (31, 0), (33, 0), (70, 64), (1100, 200), (5000, 1500), (80000, 0)])
def test_iterations_follow_the_preconditioner(bs, nb, isolated, precision, built):
    """Four iterations (the update restricts the residual for the next MAS apply)
    against PCG on the host with the same preconditioner applied by itself.  A
    stopped system is within 1e-10 |b| of its residual, 1e-8 of x (eigenvalues
    of 0.5 to about 30); a residual's last bit may round to another FP32 value
    in the mixed preconditioner: 1e-5."""
    A = block_system(nb, bs, seed=3 * nb + bs, isolated=isolated)
    b = np.random.default_rng(nb).standard_normal(A.shape[0])
    s = make_solver(bs, precision, do_hybrid_precond=False, max_iter=4)
    s.factorize(A)
    x = s.solve(b)
    its = s.get_info()["num_iterations"]
    assert 1 <= its <= 4 and (its == 4 or nb < 100)
    y, r, p, rz = np.zeros_like(b), b.copy(), 0.0, 1.0
    for _ in range(its):
        if np.linalg.norm(r) <= 1e-14 * np.linalg.norm(b):
            break
        z = s.precond(r)
        p, rz = z + (r @ z / rz) * p, r @ z
        q = A.T @ p
        alpha = rz / (p @ q)
        y, r = y + alpha * p, r - alpha * q
    assert np.linalg.norm(x - y) <= (1e-8 if precision == "fp64" else 1e-5) * np.linalg.norm(y)
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("seed", [2, 4])
def test_restart_leaves_no_residual_rounding(seed, precision, built):
    """A restarted solve is not off by what the rounding of an FP64 residual does
    to x, |A^-1 (fl(b - A x) - (b - A x))|: that is the error of any restart from
    such a residual, another one for every order of its sums.  Moduli of 1e6
    leave a residual of 5e-10 or more at a tolerance of 1e-10, so a restart cuts
    the first pass's error, of that size, by 2 (5e-10 / 1e-10)^2 = 50: a tenth of
    it is allowed."""
    import scipy.sparse.linalg as spla
    from lss import gen
    rng = np.random.Generator(np.random.PCG64(seed))
    E, _ = gen.sphere_inclusion_E(16, 16, 16, rng, E_in=1e6)
    A = gen.elasticity_cube(16, 16, 16, E)
    b = rng.standard_normal(A.shape[0])
    s = make_solver(3, precision, gmm_jump_threshold=10.0, min_subdomain_size=4)
    s.factorize(A)
    x = s.solve(b)
    assert s.get_info()["refinements"] >= 1
    s.close()
    lu = spla.splu(A.tocsc())
    wide = A.data.astype(np.longdouble)

    def residual(v):
        return b.astype(np.longdouble) - np.add.reduceat(wide * v[A.indices], A.indptr[:-1])

    y = np.zeros(len(b), np.longdouble)
    for _ in range(4):
        y = y + lu.solve(residual(y).astype(np.float64))
    z = y.astype(np.float64)
    rounding = lu.solve(((b - A @ z) - residual(z.astype(np.longdouble))).astype(np.float64))
    assert np.linalg.norm(x - z) <= 0.1 * np.linalg.norm(rounding)


@pytest.mark.parametrize("bs", [1, 2, 3])
def test_mas_apply_two_restriction_launches(bs, built):
    """MAS with more than 2048 level-1 items, whose levels above 2 are summed from
    level 2, against the CPU restatement as above (the same kind of system, the
    same bounds)."""
    import lss
    from oracle import oracle as O
    nb = 9000
    A = block_system(nb, bs, seed=nb + bs, isolated=3000)
    items = lss.coarse_space(A, bs)[0]
    assert items[1] > 2048 and len(items) > 3
    r = np.random.default_rng(nb).standard_normal(A.shape[0])
    zo = None
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-4)):
        s = make_solver(bs, precision, do_hybrid_precond=False)
        s.factorize(A)
        if zo is None:
            perm, offs = s.partition()
            zo = O.CpuSolver(A, {"block_size": bs, "do_hybrid_precond": False}, perm=perm, part_offsets=offs).precond(r)
        z = s.mas_apply(r)
        s.close()
        assert np.linalg.norm(z - zo) <= tol * np.linalg.norm(zo), precision


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("bs,nb", [(1, 600_000), (3, 295_000)])
def test_iterations_of_large_systems(bs, nb, precision, built):
    """Four iterations as above where the scalars' sums are finished by the last
    CTA (more than 311,296 rows) and the CTAs of the update and of the restriction
    take several partitions in turn (more than 19,456 and 9,728)."""
    A = block_system(nb, bs, seed=bs)
    b = np.random.default_rng(nb).standard_normal(A.shape[0])
    s = make_solver(bs, precision, do_hybrid_precond=False, max_iter=4)
    s.factorize(A)
    assert len(s.partition()[1]) - 1 > (19_456 if bs == 1 else 9_728)
    x = s.solve(b)
    assert s.get_info()["num_iterations"] == 4
    y, r, p, rz = np.zeros_like(b), b.copy(), 0.0, 1.0
    for _ in range(4):
        z = s.precond(r)
        p, rz = z + (r @ z / rz) * p, r @ z
        q = A.T @ p
        alpha = rz / (p @ q)
        y, r = y + alpha * p, r - alpha * q
    s.close()
    assert np.linalg.norm(x - y) <= (1e-8 if precision == "fp64" else 1e-5) * np.linalg.norm(y)


def test_stiff_apply_of_many_subdomains(built):
    """A_SS^-1 r on 40 stiff pieces of 1,200 DOFs with fronts of up to 440 rows:
    levels of thousands of CTAs at 64 rows, taken in chunks of 512 with more rows
    than a CTA has threads.  Bounds as above."""
    import scipy.sparse.linalg as spla
    A = block_system(20000, 3, seed=9, reach=12)
    nodes = np.concatenate([np.arange(500 * k, 500 * k + 400) for k in range(40)])
    dofs = (3 * nodes[:, None] + np.arange(3)).ravel()
    s = make_solver(3, extra={"composition": "additive"}, select_bad_dofs_from_l1_norm=False,
                    decompose_subdomains=False, expand_subdomains=False)
    s.set_problematic_dofs(dofs)
    s.factorize(A)
    info = s.get_info()
    assert info["multifrontal_subdomains"] == 40 and info["multifrontal_max_front"] > 256, info
    r = np.random.default_rng(9).standard_normal(A.shape[0])
    z = s.mas_apply(r)
    d = s.precond(r) - z
    s.close()
    x = spla.splu(A[dofs][:, dofs].tocsc()).solve(r[dofs], trans="T")
    assert np.linalg.norm(d[dofs] - x) <= 1e-12 * (np.linalg.norm(x) + np.linalg.norm(z[dofs]))
