"""Where the linear predictor's planes lie in shared memory (CKPlanes, linear.cuh):
a count of the shared-memory wavefronts of one level at 3D N=5, and the search
that the residues of its table come from.

A wavefront serves 16 lanes' 64-bit accesses as far as they fall into different
ones of 16 banks (equal addresses fall together), so an access of 16 lanes takes
as many as its fullest bank has addresses. Counted are the gradient contractions'
loads and stores, with the kernel's order of the items, and the accesses of the
per-node phase.

  python gen_planes.py            the table in linear.cuh against planes in a row
  python gen_planes.py --search [seed]   residues by simulated annealing, a minute or
                                  two a seed (the three parameters' planes are free)
"""
import math
import os
import random
import re
import sys

B, NV, ND = 6, 9, 12  # nodes per axis, elastic variables, with the parameters
YP, ZP, P = B, B * B, B ** 3
LINES = B * B
PL = P | 1  # plane pitch of the other shapes
STEP = (1, YP, ZP)


def uses(d, v):
    """ElasticPDE::ncp_uses"""
    return v >= 6 or v in ((0, 3, 5), (1, 3, 4), (2, 4, 5))[d]


PAIRS = [(d, v) for d in range(3) for v in range(NV) if uses(d, v)]
NU = len(PAIRS) // 3
PLANES = ND + len(PAIRS)


def line0(d, line):
    a, c = divmod(line, B)
    return a * ZP + c * YP if d == 0 else a * ZP + c if d == 1 else a * YP + c


def items(r, placed):
    """(component, first node of the line) of every thread in round r"""
    out = []
    for p in range(P):
        if r == 0:
            line, j = p // NU, p % NU
        elif placed and r == 1:
            line, j = p // (B * NU) * B + p % B, p // B % NU + NU
        else:
            line, j = p % LINES, p // LINES + B * r
        out.append((j, line0(PAIRS[j][0], line)))
    return out


def wavefronts(addresses):
    n = 0
    for h in range(0, len(addresses), 16):
        banks = {}
        for a in addresses[h:h + 16]:
            banks.setdefault(a % 16, set()).add(a)
        n += max(len(s) for s in banks.values())
    return n


def loads(at, placed=True):
    return sum(wavefronts([at[PAIRS[j][1]] + l0 + k * STEP[r] for j, l0 in items(r, placed)])
               for r in range(3) for k in range(B))


def stores(at, placed=True, rounds=(0, 1, 2)):
    return sum(wavefronts([at[ND + j] + l0 + k * STEP[r] for j, l0 in items(r, placed)])
               for r in rounds for k in range(B))


def per_level(at, placed=True):
    node = sum(wavefronts([at[k] + p for p in range(P)]) for k in list(range(ND, PLANES)) + list(range(NV)))
    return loads(at, placed) + stores(at, placed) + node


def in_a_row():
    return [PL * k for k in range(PLANES + 1)]


def placed_at(residue):
    at = [0]
    for k in range(1, PLANES + 1):
        a = at[-1] + P
        at.append(a + ((residue[k] - a % 16) % 16 if k < PLANES else 0))
    return at


def table():
    """the residues in linear.cuh"""
    text = open(os.path.join(os.path.dirname(os.path.abspath(__file__)), "linear.cuh")).read()
    body = re.search(r"residue\[30\] = \{(.*?)\};", text, re.S).group(1)
    return [int(x) for x in re.findall(r"\d+", re.sub(r"//.*", "", body))]


def components():
    """the gradient components' residues, each direction's stores free of conflicts:
    along x the components of one line lie side by side, along y and z as far
    apart as the lines of a plane that 16 threads cover"""
    return [j for j in range(NU)] + [YP * j % 16 for j in range(NU)] + [4 * j % 16 for j in range(NU)]


def search(seed=0, steps=40000):
    """residues of the state's planes by simulated annealing of the loads"""
    rng = random.Random(seed)
    at = [4096 * k for k in range(PLANES)]  # (apart, so that no addresses coincide)
    for k in range(NV):
        at[k] += rng.randrange(16)
    n = loads(at)
    best = (n, [at[k] % 16 for k in range(NV)])
    for i in range(steps):
        k, m = rng.randrange(NV), rng.randrange(NV)
        old = at[k], at[m]
        if k == m or rng.random() < 0.7:  # one plane moves, or two change places
            m, old = k, (at[k], at[k])
            at[k] = 4096 * k + rng.randrange(16)
        else:
            at[k], at[m] = 4096 * k + old[1] % 16, 4096 * m + old[0] % 16
        new = loads(at)
        if new <= n or rng.random() < math.exp((n - new) / (8.0 * 0.02 ** (i / steps))):
            n = new
        else:
            at[k], at[m] = old
        if n < best[0]:
            best = (n, [at[k] % 16 for k in range(NV)])
    res = [(r - best[1][0]) % 16 for r in best[1]] + [0] * (ND - NV) + components()
    return per_level(placed_at(res)), res


if __name__ == "__main__":
    if "--search" in sys.argv:
        print(*search(int(sys.argv[2]) if len(sys.argv) > 2 else 0))
    else:
        print("placed:", per_level(placed_at(table())), "in a row:", per_level(in_a_row(), placed=False))
