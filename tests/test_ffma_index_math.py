"""Index arithmetic of the FP32 FFMA MTTKRP (mttkrp_ffma.cu k_mttkrp_ffma),
restated on the CPU with the kernel's own tile arithmetic: the copies into the
X and U0 tiles, which start as NaN, the lanes' reads of them, the warps' shares
and the partials.  A read of a cell that was not copied shows as NaN, a copy
outside the tensor as an index error, a wrong place as a wrong sum."""
import os
import re

import numpy as np
import pytest

from conftest import PKG

SRC = open(os.path.join(PKG, "csrc", "mttkrp_ffma.cu")).read()
FQ, FK, FT = (int(x) for x in re.search(r"constexpr int FQ = (\d+), FK = (\d+), FT = (\d+)", SRC).groups())
NW, LDK = FT // 32, FK + 4


def plan(dims, mode, R, sms):
    others = [m for m in range(len(dims)) if m != mode]
    others = [m for m in others if dims[m] > 1] + [m for m in others if dims[m] == 1]
    P, Q, S = int(np.prod(dims[:mode])), dims[mode], int(np.prod(dims[mode + 1:]))
    rows0 = dims[others[0]]
    rtiles = -(-R // 64)
    rc = -(-R // rtiles)
    NR = 1 if rc <= 8 else 2 if rc <= 16 else 4 if rc <= 32 else 8
    TR = max(4, -(-rc // NR))
    TQ = {1: 4, 2: 8}.get(NR, 16)
    bsteps = -(-rows0 // FK)
    steps = P * S // rows0 * bsteps
    qtiles = -(-Q // FQ)
    want = max(1, (3 if TQ * TR <= 96 else 2) * sms // (qtiles * rtiles))
    chunk = -(-steps // min(want, steps))
    return dict(P=P, Q=Q, S=S, others=others, rows0=rows0, rtiles=rtiles, NR=NR, TR=TR, TQ=TQ, bsteps=bsteps,
                steps=steps, qtiles=qtiles, chunk=chunk, splits=-(-steps // chunk))


def restated(X, dims, U, mode, R, vec, sms=1):
    p = plan(dims, mode, R, sms)
    P, Q, rows0, NR, TR, TQ = p["P"], p["Q"], p["rows0"], p["NR"], p["TR"], p["TQ"]
    kq = 0 if P == 1 else 1 if vec else 2
    QL = 32 // NR
    WQ = QL * TQ
    WM = FQ // WQ
    WK, BR, TP = NW // WM, NR * TR, (TR + 3) // 4
    LDB = NR * TP * 4 + 4
    t = np.arange(FT)
    lane, warp = t & 31, t >> 5
    NC = 8 if vec else 32
    cq = (4 * lane if vec else t % FQ) if kq == 0 else (t >> 3 if vec else warp)
    ck = (warp if vec else t // FQ) if kq == 0 else (4 * (t & 7) if vec else lane)
    step = (NW if vec else FT // FQ) if kq == 0 else (FT // 8 if vec else NW)
    out = np.full((p["splits"], R, Q), np.nan)
    for cta in range(p["qtiles"] * p["splits"]):
        q0, z = cta % p["qtiles"] * FQ, cta // p["qtiles"]
        for rt in range(p["rtiles"]):
            r0 = rt * BR
            acc = np.zeros((WK, FQ, BR))
            for st in range(z * p["chunk"], min(p["steps"], (z + 1) * p["chunk"])):
                lb, lj = divmod(st, p["bsteps"])
                kc = rows0 - (p["bsteps"] - 1) * FK if lj == p["bsteps"] - 1 else FK
                A = np.full(FK * FQ if kq != 1 else FQ * LDK, np.nan)
                B = np.full(FK * LDB, np.nan)
                for th in range(FT):
                    left = Q - q0 - cq[th]
                    if kq == 0:
                        src, stride = q0 + cq[th] + Q * (lb * rows0 + lj * FK + ck[th]), step * Q
                        n = 0 if left <= 0 else (kc - ck[th] + step - 1) // step
                        dst = [(ck[th] + step * i) * FQ + cq[th] for i in range(n)]
                    else:
                        s, pb = divmod(lb, P // rows0)
                        src, stride = pb * rows0 + lj * FK + ck[th] + P * (q0 + cq[th] + Q * s), step * P
                        n = 0 if left <= 0 or ck[th] >= kc else min(NC, (left + step - 1) // step)
                        if kq == 1:
                            dst = [(cq[th] + step * i) * LDK + ck[th] for i in range(n)]
                        else:
                            swz = (ck[th] & 28) | (ck[th] & 2)
                            dst = [ck[th] * FQ + ((cq[th] + step * i) ^ swz) for i in range(n)]
                    for i, d in enumerate(dst):
                        w = 4 if vec else 1
                        assert not vec or (src + i * stride) % 4 == 0 and d % 4 == 0  # 16-byte copies are aligned
                        assert src + i * stride + w <= X.size
                        A[d: d + w] = X[src + i * stride: src + i * stride + w]
                for c in range(BR):
                    o = np.arange(kc) * LDB + c % TR // 4 * (NR * 4) + c // TR * 4 + (c % TR & 3)
                    r = min(r0 + c, R - 1)
                    B[o] = U[p["others"][0]][lj * FK + np.arange(kc) + r * rows0]
                cc, lin = np.ones(BR), lb
                for m in p["others"][1:]:
                    lin, d = divmod(lin, dims[m])
                    cc *= [U[m][d + min(r0 + c, R - 1) * dims[m]] for c in range(BR)]
                for wk in range(WK):
                    for wm in range(WM):
                        for ql in range(QL):
                            for k in range(4 * wk, kc, 4 * WK):
                                for u in range(min(4, kc - k)):
                                    if kq == 1:
                                        row = wm * WQ + ql + QL * np.arange(TQ)
                                        x = A[row * LDK + k + u]
                                    else:
                                        row, x = [], []
                                        for j in range(TQ // 4):
                                            q = wm * WQ + 4 * ql + QL * 4 * j
                                            v = A[(k + u) * FQ + (q ^ (k & 28 if kq == 2 else 0)):][:4]
                                            x += list(v[[2, 3, 0, 1]] if kq == 2 and u & 2 else v)
                                            row += range(q, q + 4)
                                    y = [B[(k + u) * LDB + 4 * (c // TR) + 4 * (c % TR // 4) * NR + (c % TR & 3)]
                                         for c in range(BR)]
                                    acc[wk][row] += np.outer(x, np.array(y) * cc)
            rows = np.arange(q0, min(q0 + FQ, Q))
            for c in range(min(BR, R - r0)):
                assert np.all(np.isnan(out[z, r0 + c, rows]))  # one writer
                out[z, r0 + c, rows] = acc.sum(0)[: rows.size, c]
    return out.sum(0).T


@pytest.mark.parametrize("dims,R", [((5, 34, 3), 3), ((33, 3, 5), 9), ((36, 130, 2), 6), ((1, 40, 7), 20), ((3, 2, 5, 4), 17),
                                    ((40, 6), 36), ((4, 1, 35), 70)])
def test_restated_kernel_matches(dims, R):
    rng = np.random.default_rng(sum(dims) + R)
    X = rng.integers(-2, 3, int(np.prod(dims))).astype(float)
    U = [rng.integers(-2, 3, d * R).astype(float) for d in dims]
    for mode in range(len(dims)):
        T = np.moveaxis(X.reshape(dims, order="F"), mode, 0).reshape(dims[mode], -1, order="F")
        kr = np.ones((1, R))
        for m in range(len(dims)):
            if m != mode:
                u = U[m].reshape(R, dims[m]).T
                kr = (u[:, None, :] * kr[None, :, :]).reshape(-1, R)
        p = plan(dims, mode, R, 1)
        run = dims[mode] if p["P"] == 1 else p["rows0"]
        for vec in ([False, True] if run % 4 == 0 else [False]):
            assert np.array_equal(restated(X, dims, U, mode, R, vec), T @ kr), (mode, vec)
