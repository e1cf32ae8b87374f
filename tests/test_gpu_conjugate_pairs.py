"""K-points whose secular problem is another's conjugate are solved once.

The candidates come from hashes; here two problems are built whose hashes
agree although they are not each other's conjugates, and every k-point must
still get its own eigenvalues and vectors.
"""
import numpy as np
import pytest

_M = (1 << 64) - 1
_A, _B, _STEP = 0xbf58476d1ce4e5b9, 0x94d049bb133111eb, 0x9e3779b97f4a7c15


def _mix(x):
    x = x ^ (x >> np.uint64(30))
    x = x * np.uint64(_A)
    x = x ^ (x >> np.uint64(27))
    x = x * np.uint64(_B)
    return x ^ (x >> np.uint64(31))


def _unshift(x, s):
    y = x
    for _ in range(64 // s + 1):
        y = x ^ (y >> np.uint64(s))
    return y


def _unmix(x):
    x = _unshift(x, 31)
    x = x * np.uint64(pow(_B, -1, 1 << 64))
    x = _unshift(x, 27)
    x = x * np.uint64(pow(_A, -1, 1 << 64))
    return _unshift(x, 30)


def _bits(x):
    return np.array([x], np.float64).view(np.uint64)


def _same_hash(h, seed):
    """A Hermitian matrix with conj(h)'s conjugate hash that is not conj(h):
    two imaginary parts of the upper triangle replaced by others of ordinary
    size, their mixed bits moved by +d and -d."""
    rng = np.random.default_rng(seed)
    n = h.shape[0]
    out = h.conj().copy()
    with np.errstate(over="ignore"):
        at = [np.array([_STEP * (c * n + r + 1) & _M], np.uint64) for r, c in ((0, 1), (2, 3))]
        re = [_mix(_bits(h[r, c].real) + a) for (r, c), a in zip(((0, 1), (2, 3)), at)]
        term = [_mix(e + _bits(h[r, c].imag)) for (r, c), e in zip(((0, 1), (2, 3)), re)]
        while True:
            d = rng.integers(1, 1 << 63, size=100000, dtype=np.uint64)
            y = [(_unmix(t + s) - e).view(np.float64)
                 for t, e, s in zip(term, re, (d, (~d) + np.uint64(1)))]
            ok = np.flatnonzero(np.all([(np.abs(v) > 0.05) & (np.abs(v) < 20.0) for v in y], axis=0))
            if ok.size:
                break
    for (r, c), v in zip(((0, 1), (2, 3)), y):
        z = complex(out[r, c].real, -v[ok[0]])  # the conjugate hash negates it
        out[r, c], out[c, r] = z, np.conj(z)
    return out


def test_constructed_matrix_has_the_same_hash_and_another_spectrum():
    rng = np.random.default_rng(1)
    a = rng.normal(size=(5, 5)) + 1j * rng.normal(size=(5, 5))
    h = a + a.conj().T
    g = _same_hash(h, 2)

    def conj_hash(m, sign):
        t = np.zeros(1, np.uint64)
        with np.errstate(over="ignore"):
            for c in range(5):
                for r in range(c + 1):
                    e = _mix(_bits(m[r, c].real + 0.0) +
                             np.array([_STEP * (c * 5 + r + 1) & _M], np.uint64))
                    t = t + _mix(e + _bits(m[r, c].imag + 0.0 if sign > 0 else 0.0 - m[r, c].imag))
        return int(t[0])

    x = np.random.default_rng(3).integers(0, 1 << 63, size=100, dtype=np.uint64)
    with np.errstate(over="ignore"):
        assert np.array_equal(_unmix(_mix(x)), x)
    assert conj_hash(g, -1) == conj_hash(h, +1) == conj_hash(h.conj(), -1)
    assert np.abs(np.linalg.eigvalsh(g) - np.linalg.eigvalsh(h)).max() > 1e-2


@pytest.mark.gpu
def test_equal_hashes_of_different_problems_are_told_apart(imago_lib, monkeypatch):
    import torch
    from imago_b200 import secular
    rng = np.random.default_rng(1)
    a = rng.normal(size=(5, 5)) + 1j * rng.normal(size=(5, 5))
    h0 = a + a.conj().T
    h = np.stack([h0, _same_hash(h0, 2), h0.conj(), _same_hash(h0, 4)])
    n, nk = 5, len(h)
    pack = lambda x: torch.as_tensor(np.stack([x[:, r, c] for c in range(n) for r in range(c + 1)], 1)
                                     .view(np.float64).reshape(nk, -1, 2), device="cuda")
    out = {"np_packed": pack(h), "ol_packed": pack(np.stack([np.eye(n, dtype=complex)] * nk)),
           "ep_packed": None}
    out["ke_packed"] = torch.zeros_like(out["np_packed"])
    monkeypatch.setattr(secular, "PAIR_MIN", 0)
    e, c = secular.secular_eigensystem(out, np.zeros(0))
    ev = secular.secular_eigenvalues(out, np.zeros(0)).cpu().numpy()
    e, c = e.cpu().numpy(), c.cpu().numpy()
    ref = np.linalg.eigvalsh(h)
    scale = np.abs(ref).max()
    # n times the rounding of a backward stable solver
    assert np.abs(e - ref).max() <= 1e-13 * scale
    assert np.abs(ev - ref).max() <= 1e-13 * scale
    assert np.abs(h @ c - c * e[:, None, :]).max() <= 1e-12 * scale
    # the one that is the first one's conjugate is still solved with it
    hs, ss = secular._secular_storage(out, np.zeros(0))
    assert list(secular._Conjugates(hs, ss).first) == [0, 1, 3]


@pytest.mark.gpu
@pytest.mark.parametrize("solve", ["secular_eigenvalues", "secular_eigensystem"])
@pytest.mark.parametrize("paired", [True, False])
def test_large_failing_overlap_names_its_k_point(imago_lib, solve, paired):
    # n > 128, factorised by torch: the message of torch.linalg.cholesky over
    # every k-point, whether or not some were left out as another's conjugate
    import torch
    from imago_b200 import secular
    rng = np.random.default_rng(6)
    n, nk = 130, 5
    a = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    a = a + a.conj().transpose(0, 2, 1)
    if paired:
        a[1] = a[0].conj()
    s = np.stack([np.eye(n, dtype=complex)] * nk)
    s[3, 6, 6] = -1.0
    with pytest.raises(torch.linalg.LinAlgError) as ref:
        torch.linalg.cholesky(torch.as_tensor(s, device="cuda"))
    assert "3" in str(ref.value) and "7" in str(ref.value)
    pack = lambda x: torch.as_tensor(np.stack([x[:, r, c] for c in range(n) for r in range(c + 1)], 1)
                                     .view(np.float64).reshape(nk, -1, 2), device="cuda")
    out = {"np_packed": pack(a), "ol_packed": pack(s), "ep_packed": None}
    out["ke_packed"] = torch.zeros_like(out["np_packed"])
    with pytest.raises(torch.linalg.LinAlgError) as err:
        getattr(secular, solve)(out, np.zeros(0))
    assert str(err.value) == str(ref.value)


@pytest.mark.gpu
def test_large_vectors_are_not_copied_where_nothing_is_paired(imago_lib):
    # n > 128: the vectors come as the triangular solve stores them, by columns
    import torch
    from imago_b200 import secular
    rng = np.random.default_rng(7)
    n, nk = 131, 2
    a = rng.normal(size=(nk, n, n)) + 1j * rng.normal(size=(nk, n, n))
    a = a + a.conj().transpose(0, 2, 1)
    pack = lambda x: torch.as_tensor(np.stack([x[:, r, c] for c in range(n) for r in range(c + 1)], 1)
                                     .view(np.float64).reshape(nk, -1, 2), device="cuda")
    out = {"np_packed": pack(a), "ol_packed": pack(np.stack([np.eye(n, dtype=complex)] * nk)),
           "ep_packed": None}
    out["ke_packed"] = torch.zeros_like(out["np_packed"])
    e, c = secular.secular_eigensystem(out, np.zeros(0))
    assert c.stride(-2) == 1
    e, c = e.cpu().numpy(), c.cpu().numpy()
    assert np.abs(a @ c - c * e[:, None, :]).max() <= 1e-11 * np.abs(e).max()
