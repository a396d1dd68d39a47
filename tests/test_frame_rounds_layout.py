"""Host-side check of the ptycho kernels' three-round transform (csrc/pt_ptycho.cu).

A det x det frame passes through shared memory as rows (k1, j) of QB values qb
whose 16-byte slots are XORed with k1 & 7: j = qa RT + rt after the first round
and v1 RT + k2 after the second, which works in place.  This restates the index
maps for every detector size and checks that the layout is a bijection, that
each warp access takes the minimum number of shared-memory wavefronts (32 banks
of 4 bytes), that the second round reads and writes the same slots, and that the
rounds compute B[u][v] = sum A[r][q] w^(u r + v q).  No GPU is needed."""
import numpy as np
import pytest

DETS = [16, 32, 64, 128]


def sizes(det):
    qb = 32 if det == 128 else 16
    return qb, det // qb, det // 16          # QB, QA, RT


def at(det, k1, j, qb):
    QB, QA, RT = sizes(det)
    return (k1 * QA * RT + j) * QB + 2 * ((qb >> 1) ^ (k1 & 7)) + (qb & 1)


def wavefronts(byte_addrs, size):
    banks = {}
    for a in byte_addrs:
        for o in range(0, size, 4):
            word = (a + o) // 4
            banks.setdefault(word % 32, set()).add(word)
    return max(len(s) for s in banks.values())


@pytest.mark.parametrize("det", DETS)
def test_rounds_layout(det):
    QB, QA, RT = sizes(det)
    k1, j, qb = np.meshgrid(np.arange(16), np.arange(QA * RT), np.arange(QB), indexing="ij")
    assert np.array_equal(np.sort(at(det, k1, j, qb).ravel()), np.arange(det * det))
    lanes = np.arange(32)
    # round 1 writes (8 bytes): 32 consecutive lines (q fastest), one k1
    for first in range(0, det * RT, 32):
        q, rt = (first + lanes) % det, (first + lanes) // det
        if det * RT < 32 and first:
            break
        for k in range(16):
            assert wavefronts(8 * at(det, k, (q // QB) * RT + np.minimum(rt, RT - 1), q % QB), 8) <= 2
    # round 2 reads and writes (8 bytes): 32 consecutive (k1, qb), one row j
    for first in range(0, 16 * QB, 32):
        a, b = (first + lanes) // QB, (first + lanes) % QB
        for row in range(QA * RT):
            assert wavefronts(8 * at(det, a, row, b), 8) == 2
    # round 3 reads (16 bytes): 32 consecutive u of one v1, slot s ^ (k1 & 7)
    for first in range(0, det, 32):
        u = (first + lanes) % det
        for v1 in range(QA):
            row = ((u % 16) * QA * RT + v1 * RT + u // 16) * QB
            for s in range(QB // 2):
                need = 4 if det >= 32 else 2          # 16 distinct rows of 16 bytes at det 16
                assert wavefronts(8 * row + 16 * (s ^ (u % 16 & 7)), 16) <= need


@pytest.mark.parametrize("det", DETS)
@pytest.mark.parametrize("sign", [-1, 1])
def test_rounds_compute_the_dft(det, sign):
    QB, QA, RT = sizes(det)
    rng = np.random.default_rng(det)
    A = rng.standard_normal((det, det)) + 1j * rng.standard_normal((det, det))
    w = lambda x: np.exp(sign * 2j * np.pi * x / det)  # noqa: E731
    ex = np.full(det * det, np.nan, complex)
    k = np.arange(16)
    for q in range(det):                                # round 1: line (q, rt)
        for rt in range(RT):
            line = A[rt + RT * k, q]
            X = np.exp(sign * 2j * np.pi * np.outer(k, k) / 16) @ line * w(rt * k)
            ex[at(det, k, (q // QB) * RT + rt, q % QB)] = X
    f = 0.7 - 0.2j
    for k1 in range(16):                                # round 2: (k1, qb), in place
        for qb in range(QB):
            a = ex[at(det, k1, np.arange(QA * RT), qb)].reshape(QA, RT)
            a = a @ np.exp(sign * 2j * np.pi * np.outer(np.arange(RT), np.arange(RT)) / RT)
            a = np.exp(sign * 2j * np.pi * np.outer(np.arange(QA), np.arange(QA)) / QA) @ a
            ex[at(det, k1, np.arange(QA * RT), qb)] = (a * (w(qb * np.arange(QA)) * f)[:, None]).ravel()
    B = np.empty((det, det), complex)
    m = np.arange(QB)
    for u in range(det):                                # round 3: row (u, v1)
        for v1 in range(QA):
            row = ex[at(det, u % 16, v1 * RT + u // 16, m)]
            B[u, v1 + QA * m] = np.exp(sign * 2j * np.pi * np.outer(m, m) / QB) @ row
    ref = f * (np.fft.fft2(A) if sign < 0 else np.fft.ifft2(A) * det * det)
    assert np.allclose(B, ref, rtol=0, atol=1e-10 * np.abs(ref).max())
