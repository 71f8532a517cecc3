"""The builds at the sizes where their tiles, panels and blocks end, against plain torch (B200)."""

from __future__ import annotations

import numpy as np
import pytest

from hafnium_b200 import _lib
from hafnium_b200.errors import InputError
from hafnium_b200.molecule import water_cluster
from tests.test_gpu_coulomb import hydrogen_tables, hydrogens

pytestmark = pytest.mark.gpu
EPS = 2.3e-16


# column tiles of 32, 48, 64 and 80, one column more than each, several of them; odd n
@pytest.mark.parametrize("columns", [1, 16, 17, 32, 33, 48, 49, 64, 65, 80, 81, 96, 97, 160, 161])
@pytest.mark.parametrize("signed", [False, True])
def test_exchange_of_every_column_tile(columns, signed):
    import torch

    n, n_aux = 129, 37
    two_body = hydrogens(n, n_aux)
    gen = torch.Generator().manual_seed(columns)
    c = torch.randn((n, columns), dtype=torch.float64, generator=gen).cuda()
    w = torch.randn(columns, dtype=torch.float64, generator=gen).cuda() if signed else None
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    b = two_body.orbital_tensor(eye, eye)
    x = torch.einsum("quv,vi->qui", b, c)
    expected = torch.einsum("qui,qvi->uv", x if w is None else x * w, x)
    # two sums of n, then n_aux columns products: each errs by at most its length times eps times
    # the sum of its absolute terms
    ax = torch.einsum("quv,vi->qui", b.abs(), c.abs())
    size = torch.einsum("qui,qvi->uv", ax if w is None else ax * w.abs(), ax)
    got = two_body.exchange_factored(c, w)
    assert float(((got - expected).abs() / ((2 * n + n_aux * columns) * EPS * size)).max()) < 1.0


# X's rows in several chunks (4 GB in FP64, 2 GB in split BF16, half as many rows with a signed factor): K is
# then added up chunk by chunk
@pytest.mark.parametrize("signed", [False, True])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_BF16X3])
def test_exchange_in_several_chunks_of_rows(signed, precision):
    import torch

    n, n_aux, columns = 1030, 600, 1000
    two_body = hydrogens(n, n_aux)
    gen = torch.Generator().manual_seed(columns)
    c = torch.randn((n, columns), dtype=torch.float64, generator=gen).cuda()
    w = torch.randn(columns, dtype=torch.float64, generator=gen).cuda() if signed else None
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    b = two_body.orbital_tensor(eye, eye)
    expected, size = torch.zeros_like(eye), torch.zeros_like(eye)
    for q in range(0, n_aux, 50):
        x, ax = b[q:q + 50] @ c, b[q:q + 50].abs() @ c.abs()
        expected += torch.einsum("qui,qvi->uv", x if w is None else x * w, x)
        size += torch.einsum("qui,qvi->uv", ax if w is None else ax * w.abs(), ax)
    for _ in range(2):
        got = two_body.exchange_factored(c, w, precision)
        error = (got - expected).abs()
        if precision == _lib.PREC_FP64:  # two sums of n, then n_aux columns products
            assert float((error / ((2 * n + n_aux * columns) * EPS * size)).max()) < 1.0
        else:
            # 16 bits of each factor, and each addition of 16 products to a 32-bit sum truncates by up to 2^-23: a
            # chunk's 450 rows of 1000 columns in three products, split twelve ways, are 7000 additions, 8e-4; a
            # signed sum against its parts
            scale = expected if w is None else two_body.exchange_factored(c, w.abs())
            assert float(error.max()) <= 1e-3 * float(scale.abs().max())
        assert torch.equal(got, got.T)


def test_a_context_without_a_word_of_mapped_memory():
    """The page of words that kernels write for the host has 1024 of them; later contexts copy, and their J is
    built in two passes."""
    import torch

    n, n_aux = 129, 300
    c = torch.randn((n, 20), dtype=torch.float64, generator=torch.Generator().manual_seed(n)).cuda()
    d = c @ c.T
    contexts = [_lib.Context() for _ in range(1026)]
    results = []
    for context in (contexts[0], contexts[-1]):
        context.upload(*hydrogen_tables(n, n_aux))
        context.build()
        j, k, k16 = torch.empty_like(d), torch.empty_like(d), torch.empty_like(d)
        before = context.stats()["kernel_launches"]
        context.coulomb_device(d, j)
        launches = context.stats()["kernel_launches"] - before
        context.exchange_device(d, k)
        context.exchange_device(d, k16, _lib.PREC_BF16X3)
        f = context.density_factor_device(d, n)
        results.append((launches, j, k, k16, f))
        with pytest.raises(InputError, match="semidefinite"):
            context.density_factor_device(-d, n)
    (first, j0, *others), (last, j1, *same) = results
    assert (first, last) == (1, 4)
    assert float((j0 - j1).abs().max()) < 2.3e-16 * (n * n + n_aux) * float(j0.abs().max())
    for x, y in zip(others, same):
        assert torch.equal(x, y)
    for context in contexts:
        context.close()


# one panel and several, rows of L in shared memory, ranks that end inside and at the end of a panel
@pytest.mark.parametrize("n,rank", [(1, 1), (2, 1), (33, 33), (160, 40), (161, 161), (300, 70), (300, 95), (900, 64),
                                    (900, 200)])
def test_density_factor_across_panels(n, rank):
    import torch

    two_body = hydrogens(n, 3)
    gen = torch.Generator().manual_seed(n + rank)
    c = torch.randn((n, rank), dtype=torch.float64, generator=gen).cuda() / np.sqrt(n)
    d = c @ c.T
    f = two_body.context.density_factor_device(d, n)
    assert rank <= f.shape[1] <= n
    # a Cholesky factor reproduces each element to its length times eps of the diagonal's size, and the
    # remainder it stops at is 1e-14 of the largest diagonal element
    bound = ((rank + 2) * EPS + 1e-14) * float(d.diagonal().max()) * 4
    assert float((f @ f.T - d).abs().max()) < bound


# the narrowest panels with their rows in shared memory and the first without, the largest n whose diagonal
# is there too and the first without; several panels each
@pytest.mark.parametrize("n,rank", [(2560, 33), (2560, 70), (2561, 33), (2561, 70), (22528, 40), (22529, 40)])
def test_density_factor_of_large_matrices(n, rank):
    import torch

    context = _lib.Context()
    context.upload(hydrogen_tables(n, 1)[0])
    gen = torch.Generator().manual_seed(n + rank)
    c = torch.randn((n, rank), dtype=torch.float64, generator=gen).cuda() / np.sqrt(n)
    d = c @ c.T
    f = context.density_factor_device(d, rank + 30)
    assert rank <= f.shape[1] <= rank + 30
    # as above
    bound = ((rank + 2) * EPS + 1e-14) * float(d.diagonal().max()) * 4
    assert max(float((part @ f.T - rows).abs().max()) for part, rows in zip(f.split(2048), d.split(2048))) < bound


# blocks of 64: one, a ragged one, several, with and without a remainder
@pytest.mark.parametrize("n_aux", [1, 63, 64, 65, 127, 128, 130, 193, 256, 257, 321, 450])
def test_the_fit_at_the_factors_block_edges(n_aux):
    import torch

    two_body = hydrogens(20, n_aux)
    eye = torch.eye(20, dtype=torch.float64, device="cuda")
    b = two_body.orbital_tensor(eye, eye).reshape(n_aux, -1)
    metric = torch.as_tensor(two_body.context.metric()).cuda()
    three = torch.as_tensor(two_body.context.three_center()).cuda().reshape(n_aux, -1)
    low = torch.linalg.cholesky(metric)
    expected = torch.linalg.solve_triangular(low, three, upper=False)  # one shell per function: the same order
    condition = float(torch.linalg.cond(metric))
    bound = 8 * n_aux * EPS * condition * float(expected.abs().max())
    assert float((b - expected).abs().max()) < bound


# the purification in one CTA (up to 112 functions) and in launches past it, n odd and at the edge
@pytest.mark.parametrize("waters,basis", [(1, "sto-3g"), (1, "cc-pvdz"), (15, "sto-3g"), (16, "sto-3g"), (17, "sto-3g")])
def test_batched_scf_at_the_purification_sizes(waters, basis):
    from hafnium_b200.batch import solve_batch
    from hafnium_b200.scf import DeviceHamiltonian, atomic_density_guess, solve_rhf

    mols = [water_cluster(waters, s) for s in (1, 2)]
    batch = solve_batch(mols, basis, setup_threads=2, retry_failed=False)
    for mol, energy, state in zip(mols, batch.energies, batch.states):
        ham = DeviceHamiltonian.build(mol, basis, "def2-universal-jkfit")
        ref = solve_rhf(ham, guess=atomic_density_guess(mol, basis))
        assert state == "converged"
        # both stop at a commutator of 1e-6 or less, and the energy errs by its square
        assert abs(energy - ref.energy) < 1e-8
