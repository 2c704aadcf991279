"""FP64 products on the integer pipes with operands and factors of every kind:
zeros of both signs, subnormals, short values, values and factors near the ends
of the range.  Diagonal systems, whose solution is one product a row, are the
IEEE products bit for bit through every FP64 kernel that scales its rows so."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _values(shape, seed):
    rng = np.random.default_rng(seed)
    d = rng.normal(size=shape)
    kind = rng.integers(0, 12, size=shape)
    d[kind == 0] = 0.
    d[kind == 1] = -0.
    d[kind == 2] = 1.
    d[kind == 3] *= 1e-310
    d[kind == 4] *= 1e-229
    d[kind == 5] *= 1e229
    d[..., : shape[-1] // 3] *= np.where(rng.random(shape[:-1] + (1,)) < .5, 0., 1.)  # quiet regions
    d.reshape(-1, shape[-1])[0, np.abs(d.reshape(-1, shape[-1])[0]) > 1e100] = 1.  # one system cannot overflow
    return d


def _same(got, want):
    assert np.array_equal(got, want)
    assert np.array_equal(np.signbit(got), np.signbit(want))


FACTORS = [2. / 3, 1. / 3, -3., 1e-25, -1.1e25, 1.7e74, 1.3e-80]


@pytest.mark.parametrize("b", FACTORS)
@pytest.mark.parametrize("nsys,n", [(3, 100), (200, 41), (200000, 33)])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("chunks", [1, 2])
def test_plan(cuda, b, nsys, n, strided, chunks):
    import ntk

    d = _values((nsys, n), n)
    g = 1. / np.float64(b)
    with np.errstate(over="ignore", under="ignore"):
        want = d * g
    keep = np.isfinite(want).all(axis=1)  # an overflow spreads to other rows (0 * inf)
    assert keep.any()
    t = torch.from_numpy(d.T.copy() if strided else d.copy()).to(cuda)
    with ntk.Plan(n, nsys, (b, 0., 0., b, 0., 0., b)) as p:
        p.set_tuning(f64_chunks=chunks)
        if strided:
            p.solve_strided(t, t, nsys, nsys, 1, 0, nsys)
        else:
            p.solve(t)
    got = t.cpu().numpy().T if strided else t.cpu().numpy()
    # the sweeps add -w x = -+0 to each row's product: only the sign of a zero can change
    nz = want[keep] != 0
    _same(got[keep][nz], want[keep][nz])
    assert (got[keep][~nz] == 0).all()


@pytest.mark.parametrize("b", FACTORS)
def test_batch(cuda, b):
    import ntk

    n = np.array([40, 700, 3000, 512, 17], dtype=np.int32)
    row = np.array([0., b, 0.])
    d = _values((int(n.sum()),), 2)
    d[np.abs(d) > 1e100] = 1.5
    want = d * (1. / np.float64(b))
    t = torch.from_numpy(d).to(cuda)
    with ntk.UnevenBatch(n, np.tile(row, (5, 1)), np.tile(row, (5, 2, 1)), np.tile(row, (5, 2, 1))) as batch:
        batch.solve(t)
    got = t.cpu().numpy()
    nz = want != 0
    _same(got[nz], want[nz])
    assert (got[~nz] == 0).all()


@pytest.mark.parametrize("n", [33, 257])
@pytest.mark.parametrize("axis", [1, 2])
def test_the_same_solution_whatever_the_batch(cuda, n, axis):
    """One thread per system: the choice between the integer and the FP64
    product by the number of systems changes no bit."""
    import ntk

    many = 130000
    d = torch.from_numpy(_values((1, many, n), 5)).to(cuda).nan_to_num_()
    d[d.abs() > 1e100] = 2.
    few = d[:, :70].contiguous()
    if axis == 1:
        d, few = d.transpose(1, 2).contiguous(), few.transpose(1, 2).contiguous()
    a, b = torch.empty_like(d), torch.empty_like(few)
    with ntk.Plan(n, 0, (1., 2., .25, 1., .25, 2., 1.)) as p:
        p.set_tuning(f64_chunks=1)
        p.compact_deriv(d, a, axis, .01)
        p.compact_deriv(few, b, axis, .01)
    a = a[:, :, :70] if axis == 1 else a[:, :70]
    assert torch.equal(a, b)
