"""CPU model of the row form of the x / z pass (test infrastructure).

The tableau's column of generator g evolves under gates independently of
every other column, so the gates of a whole program run first (``raw_rows``):
every measurement dumps its row x_q over the 2n initial generators (S: the
stabilizer half, T: the destabilizer half), and from then on also owns a
column of its own -- the generator Z_q it puts into the tableau -- whose
entries in later rows replace the pivot column's.  ``eliminate`` then walks
the measurements in order on those rows alone: a random one (S != 0, pivot p)
becomes an update of the rows after it,
    S_i += a F_S, T_i += a F_T (a = S_i[p], F = -e S_j, -e T_j without p),
    T_i[p] = e a, S_i[p] = the raw entry of row i in measurement j's column.
RESET's z_q row and an N1's x_q and z_q rows are rows of the same kind whose
stabilizer half only is needed; ``after`` says how many measurements' updates
they take.

Phases.  Odd d: with X^x Z^z = omega^(-xz/2) W(x, z) the product of commuting
W is W of the sum and H, CNOT change no phase; P and the Paulis add a linear
form of the column, kept as one more raw column (the constant column), and
the generators' phases V_g follow the same update as a row.  d = 2: the rows
are Paulis i^k prod_g X_g^(S_g) Z_g^(T_g) whose exponent k follows the gates
(a product of rows adds twice the parity of T . S') and the update (below).
"""
from __future__ import annotations

import numpy as np


class Rows:
    def __init__(self, n, d):
        self.n, self.d = n, d
        self.meas = []    # (x row, constant or sign, reset)
        self.extra = []   # (row, updates that it takes, owner): S half and raw columns


def raw_rows(n, d, words):
    """words: (op, q, t) device instructions; gates 1..10, 14 M, 16 RESET, 17 N1."""
    nm = sum(op in (14, 16) for op, _, _ in words)
    cols = 2 * n + nm
    X, Z = np.zeros((n, cols), np.int64), np.zeros((n, cols), np.int64)
    for k in range(n):
        Z[k, k] = 1
        X[k, n + k] = 1
    kx, kz = np.zeros(n, np.int64), np.zeros(n, np.int64)
    half = (d + 1) // 2
    out, mord, nord = Rows(n, d), 0, 0

    def mul2(a, b):  # parity of Z exponents of row a against X exponents of row b
        return int((a[n:2 * n] & b[:n]).sum()) & 1

    for op, q, t in words:
        if op in (14, 16):
            out.meas.append((X[q].copy(), int(kx[q]), op == 16))
            Z[q, 2 * n + mord] = 1
            mord += 1
            if op == 16:
                out.extra.append((Z[q].copy(), mord, ("reset", mord - 1)))
        elif op == 17:
            out.extra.append((X[q].copy(), mord, ("nx", nord)))
            out.extra.append((Z[q].copy(), mord, ("nz", nord)))
            nord += 1
        elif d == 2:
            if op in (1, 2):
                kx[q] += 2
            elif op in (3, 4):
                kz[q] += 2
            elif op in (5, 6):
                X[q], Z[q] = Z[q].copy(), X[q].copy()
                kx[q], kz[q] = kz[q], kx[q]
            elif op in (7, 8):
                kz[q] += kx[q] + (3 if op == 7 else 1) + 2 * mul2(Z[q], X[q])
                Z[q] ^= X[q]
            else:
                kx[t] += kx[q] + 2 * mul2(X[q], X[t])
                kz[q] += kz[t] + 2 * mul2(Z[q], Z[t])
                X[t] ^= X[q]
                Z[q] ^= Z[t]
            kx %= 4
            kz %= 4
        else:
            if op == 1:
                kx[q] += 1
            elif op == 2:
                kx[q] -= 1
            elif op == 3:
                kz[q] += 1
            elif op == 4:
                kz[q] -= 1
            elif op == 5:
                X[q], Z[q] = -Z[q], X[q].copy()
                kx[q], kz[q] = -kz[q], kx[q]
            elif op == 6:
                X[q], Z[q] = Z[q].copy(), -X[q]
                kx[q], kz[q] = kz[q], -kx[q]
            elif op == 7:
                Z[q] += X[q]
                kz[q] += kx[q] - half
            elif op == 8:
                Z[q] -= X[q]
                kz[q] += half - kx[q]
            else:
                s = 1 if op == 9 else -1
                X[t] += s * X[q]
                Z[q] -= s * Z[t]
                kx[t] += s * kx[q]
                kz[q] -= s * kz[t]
            X %= d
            Z %= d
            kx %= d
            kz %= d
    return out


def eliminate(rows):
    """Trace records: per measurement (kind, pivot, exponent, phase, factor
    row over the stabilizers, z_q row or None); and the N1 rows (x, z)."""
    n, d = rows.n, rows.d
    V = np.zeros(n, np.int64)
    ops, recs = [], []

    def apply(S, T, raw, k, op):
        """One update on a row; T None: the stabilizer half only.  d = 2: k the sign exponent."""
        p, e, FS, FT, j, tp = op
        a = int(S[p])
        om = int(raw[2 * n + j])
        if a:
            S = (S + a * FS) % d
            if T is not None:
                T = (T + a * FT) % d
        if d == 2 and T is not None and a:
            # S here is the row after the update; FS, FT hold no bit p
            k += 2 * (int((S * FT).sum() - S[p] * FT[p]) & 1) + tp + 2 * om
        S[p] = om
        if T is not None:
            T[p] = e * a % d
        return S, T, k

    for j, (raw, k, reset) in enumerate(rows.meas):
        S, T = raw[:n].copy(), raw[n:2 * n].copy()
        for op in ops:
            S, T, k = apply(S, T, raw, k, op)
        nz = np.nonzero(S)[0]
        if len(nz):
            p = int(nz[0])
            e = pow(int(S[p]), d - 2, d) if d > 2 else 1
            FS, FT = (-e * S) % d, (-e * T) % d
            FW = (-S) % d
            FS[p] = FT[p] = FW[p] = 0
            if d == 2:
                tp = int((S * T).sum()) & 1
                V = (V + FS * V[p]) % 2
                V[p] = ((k + tp) // 2) & 1
                assert (k + tp) % 2 == 0
                ops.append((p, 1, FS, FT, j, tp))
            else:
                V = (V + FS * V[p]) % d
                V[p] = k
                ops.append((p, e, FS, FT, j, 0))
            recs.append(["rand", p, e, 0, FW, None])
        else:
            a = (2 * ((k // 2 + int((T * V).sum())) & 1)) if d == 2 else int((T * V).sum() - k) % d
            recs.append(["det", 0, 1, a, T, None])
    order = [op[4] for op in ops]
    n1 = {}
    for raw, after, who in rows.extra:
        S = raw[:n].copy()
        for op, j in zip(ops, order):
            if j < after:
                S, _, _ = apply(S, None, raw, 0, op)
        if who[0] == "reset":
            recs[who[1]][5] = S
        else:
            n1[who] = S
    return recs, n1


def replay(recs, n, d, outcome):
    """Records of one noiseless shot from the trace: outcome(k) the draw of measurement k."""
    delta = np.zeros(n, np.int64)
    out = []
    for k, (kind, p, e, a, row, zrow) in enumerate(recs):
        if kind == "rand":
            dp = int(delta[p]) * e % d
            delta = (delta + row * dp) % d
            m = outcome(k)
            delta[p] = (-m) % d
        else:
            s = int((row * delta).sum())
            m = ((a // 2 + s) & 1) if d == 2 else (-(a + s)) % d
        if zrow is not None:
            delta = (delta + m * zrow) % d
        out.append(m | (128 if kind == "det" else 0))
    return np.array(out, np.uint8)
