"""GPU: one product of the INT8 update at a time (through the library's C++ symbols: no public
call runs one alone), against exact integers.  The panels' entries are numbers whose seven
digits are exact, so that what is left is the levels past 7, the last unit and the roundings:
tight enough that a lost digit plane, level or carry shows."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

UPDATE = "_ZN2hs19launch_split_updateEP8hs_ctx_sPdiiiPvP11CUstream_st"
UPDATE_BYTES = "_ZN2hs18split_update_bytesEiii"
STEP = "_ZN2hs25launch_split_inverse_stepEP8hs_ctx_sPdiPKdS2_PvP11CUstream_stS7_RA2_P10CUevent_st"
STEP_BYTES = "_ZN2hs19split_inverse_bytesEi"
_P, _I = ctypes.c_void_p, ctypes.c_int


def _symbol(hs, name, restype, *argtypes):
    fn = getattr(hs._lib.load(), name)
    fn.restype, fn.argtypes = restype, argtypes
    return fn


def _rows(kind, n, K, seed):
    """n rows of K integers below 2^54 in size, in units of 2^-54 times 2^shift a row."""
    rng = np.random.default_rng(seed)
    sign = rng.choice([-1, 1], (n, K))
    if kind == "random":
        v = rng.integers(0, 1 << 52, (n, K)) << 2
    elif kind == "spread":  # entries of 1 to 52 bits
        v = (rng.integers(0, 1 << 52, (n, K)) >> rng.integers(0, 52, (n, K))) << 2
    else:  # digits 127 and -128 throughout; whole rows of one sign
        v = np.where(rng.random((n, K)) < 0.5, 0x7F3A7F7F7F7F7C, 0x7E808080808080) >> 1
        sign[: n // 2] = 1
    shift = rng.integers(-300, 300, n) if kind == "spread" else np.zeros(n, dtype=np.int64)
    return (sign * v).astype(np.int64), shift


def _values(v, shift):
    return torch.from_numpy(np.ldexp(v.astype(np.float64), shift[:, None] - 54)).cuda()


def _scale(v):
    """The kernel's exponent of a row's scale, without the row's shift: |x| 2^-e <= 0.497."""
    f, e = np.frexp(np.abs(v).max(axis=1).astype(np.float64) * 2.0 ** -54)
    return e + 1 + (f >= (1 + 253 / 256) / 2)


def _exact(a, b):
    """a b^T of integers below 2^54, as Python integers: three 18-bit limbs each, whose products'
    sums stay below 2^53."""
    def limbs(v):
        out = []
        for _ in range(2):
            low = ((v + (1 << 17)) & ((1 << 18) - 1)) - (1 << 17)
            out.append(low)
            v = (v - low) >> 18
        return [torch.from_numpy(x.astype(np.float64)).cuda() for x in out + [v]]

    total = 0
    for i, x in enumerate(limbs(a)):
        for j, y in enumerate(limbs(b)):
            total = total + ((x @ y.T).cpu().numpy().astype(np.int64).astype(object) << (18 * (i + j)))
    return total


def _check(got, a, b, sa, sb, K, sign, mask=None):
    """got (float64, from zero) = sign a b^T within 2^-53 of itself plus, in units of the two
    scales, K products' levels past 7 (5.02 x 2^-66 each) and half of the last unit 2^-56."""
    exact = sign * _exact(a, b)
    got = np.ldexp(got.cpu().numpy(), 108 - sa[:, None] - sb[None, :])
    err = np.array([[abs(int(g) - x) for g, x in zip(gr, xr)] for gr, xr in zip(got, exact)], dtype=np.float64)
    unit = np.ldexp(1.0, (_scale(a)[:, None] + _scale(b)[None, :]) + 108)
    bound = 2.0 ** -53 * np.abs(exact.astype(np.float64)) + unit * (K * 5.02 * 2.0 ** -66 + 2.0 ** -57)
    if mask is not None:
        err, bound = err[mask], bound[mask]
    assert np.all(err <= bound), (err / bound).max()


@pytest.mark.parametrize("kind", ["random", "spread", "ends"])
@pytest.mark.parametrize("bsz,panels,nb,k,col", [(256, 1, 4, 0, 1), (256, 1, 5, 1, 3), (256, 2, 5, 0, 2),
                                                 (256, 2, 6, 1, 4), (128, 2, 6, 0, 2), (128, 2, 7, 1, 4)])
def test_trailing_update(hs, ctx, kind, bsz, panels, nb, k, col):
    ctx.set_problem(nb * bsz, bsz)
    row0, K = k + panels, panels * bsz
    v, shift = _rows(kind, (nb - row0) * bsz, K, 7 * nb + bsz + panels)
    P = _values(v, shift)
    A = torch.zeros(hs.packed_size(nb * bsz, bsz), dtype=torch.float64, device="cuda")

    def block(i, j):
        s = hs.block_id(i, j, nb) * bsz * bsz
        return A[s:s + bsz * bsz].view(bsz, bsz)

    for i in range(row0, nb):
        for p in range(panels):
            block(i, k + p).copy_(P[(i - row0) * bsz:(i - row0 + 1) * bsz, p * bsz:(p + 1) * bsz])
    before = A.clone()
    ws = torch.empty(_symbol(hs, UPDATE_BYTES, ctypes.c_size_t, _I, _I, _I)(nb, bsz, panels), dtype=torch.uint8,
                     device="cuda")
    st = _symbol(hs, UPDATE, _I, _P, _P, _I, _I, _I, _P, _P)(
        ctx.handle, A.data_ptr(), k, panels, col, ws.data_ptr(), ctx.stream.cuda_stream)
    assert st == 0 and ctx.take_info() == -1
    n = (nb - col) * bsz
    C = torch.zeros((n, n), dtype=torch.float64, device="cuda")
    for j in range(col, nb):
        for i in range(j, nb):
            C[(i - col) * bsz:(i - col + 1) * bsz, (j - col) * bsz:(j - col + 1) * bsz] = block(i, j)
            block(i, j).zero_()
    assert torch.equal(A, before)  # nothing else is written
    assert not C.triu(1).any()
    v, shift = v[(col - row0) * bsz:], shift[(col - row0) * bsz:]
    _check(C, v, v, shift, shift, K, -1, np.tril(np.ones((n, n), dtype=bool)))


@pytest.mark.parametrize("kind", ["random", "spread", "ends"])
@pytest.mark.parametrize("nb,k", [(3, 0), (3, 1), (3, 2)])
def test_step_of_the_inverse(hs, ctx, kind, nb, k):
    """S_rc -= L_rk W_c for the rows below, L_rc += W_r^T W_c, after column k of L is cleared."""
    bsz = 256
    bb = bsz * bsz
    ctx.set_problem(nb * bsz, bsz)
    wv, wshift = _rows(kind, (k + 1) * bsz, bsz, 11 * nb + k)  # columns of W, one after the other
    W = torch.stack([w.T.contiguous() for w in _values(wv, wshift).view(k + 1, bsz, bsz)])
    lv, lshift = _rows(kind, (nb - k - 1) * bsz, bsz, 13 * nb + k)
    L = torch.zeros(hs.packed_size(nb * bsz, bsz), dtype=torch.float64, device="cuda")
    first = hs.block_id(k, k, nb)
    L[first * bb:(first + 1) * bb] = 3.0
    if k + 1 < nb:
        L[(first + 1) * bb:(first + nb - k) * bb] = _values(lv, lshift).reshape(-1)
    S = torch.zeros(nb * (nb + 1) // 2 * bb, dtype=torch.float64, device="cuda")
    ws = torch.empty(_symbol(hs, STEP_BYTES, ctypes.c_size_t, _I)(nb), dtype=torch.uint8, device="cuda")
    side, events = torch.cuda.Stream(), [torch.cuda.Event(), torch.cuda.Event()]
    for e in events:
        e.record(ctx.stream)
    done = (_P * 2)(*[e.cuda_event for e in events])
    st = _symbol(hs, STEP, _I, _P, _P, _I, _P, _P, _P, _P, _P, _P)(
        ctx.handle, L.data_ptr(), k, W.data_ptr(), S.data_ptr(), ws.data_ptr(), ctx.stream.cuda_stream,
        side.cuda_stream, done)
    torch.cuda.synchronize()
    assert st == 0 and ctx.take_info() == -1
    for r in range(nb):
        for c in range(r + 1):
            w = slice(c * bsz, (c + 1) * bsz)
            got = S[(r * (r + 1) // 2 + c) * bb:][:bb].view(bsz, bsz)
            if r > k and c <= k:
                rows = slice((r - k - 1) * bsz, (r - k) * bsz)
                _check(got, lv[rows], wv[w], lshift[rows], wshift[w], bsz, -1)
            else:
                assert not got.any()
            got = L[hs.block_id(r, c, nb) * bb:][:bb].view(bsz, bsz)
            if r <= k:
                rows = slice(r * bsz, (r + 1) * bsz)
                lower = np.tril(np.ones((bsz, bsz), dtype=bool)) if r == c else None
                _check(got, wv[rows], wv[w], wshift[rows], wshift[w], bsz, 1, lower)
                assert r != c or not got.triu(1).any()
            else:
                assert not got.any()
