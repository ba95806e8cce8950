"""Mechanisms as large as the kernels' shared memory: GRI-3.0's species with its reactions repeated, each copy with other
pre-exponential factors, and for the last bytes a few reactions of the smallest footprint."""
import copy

SMEM = 232448  # shared memory a block can have
ORDER = {'simple': 0, 'three-body': 1, 'Lindemann': 2, 'Troe': 3}


def mechanism(repeats, small=0):
    """GRI-3.0's species, `repeats` reactions taken from its list over and over, and `small` irreversible ones."""
    from spitfire_gb300.mechanism import ChemicalMechanismSpec
    md = copy.deepcopy(ChemicalMechanismSpec.bundled('methane-gri30').mech_data)
    base = [list(r) for r in md['reactions']]
    rx = []
    for k in range(repeats):
        r = list(base[k % len(base)])
        r[4] = r[4] / (1. + k // len(base))
        if len(r) > 9:
            r[9] = r[9] / (1. + k // len(base))
        rx.append(tuple(r))
    rx += [('simple', {'H': 1.}, {'O': 1.}, False, 1e-3 * (1 + k), 0., 0.) for k in range(small)]
    rx.sort(key=lambda r: ORDER[r[0]])
    md['reactions'] = rx
    return ChemicalMechanismSpec(mech_data=md)


def search(value, target, lo, hi):
    """The largest k in [lo, hi] whose value(k), increasing in k, is at most `target`."""
    while lo < hi:
        mid = (lo + hi + 1) // 2
        lo, hi = (mid, hi) if value(mid) <= target else (lo, mid - 1)
    return lo


def plain_need(spec):
    """(right-hand side, Jacobian) shared memory in bytes of one narrow group in the plain layout: the mechanism's tables with
    FP64 rate constants alone, and every scratch array in a place of its own."""
    a = spec.griffon._rec.arrays()
    rx = spec.griffon._rec.reactions
    ns, nr = len(a['mw']), len(rx)
    even = lambda k: k + (k & 1)
    last = spec.griffon._rec.species[-1]
    n_fall = sum(r['kind'] >= 3 for r in rx)
    lists = [[set(r[k]) for r in rx] for k in ('reactants', 'products', 'efficiencies')]
    nreac, nprod, ntb = (sum(len(x) for x in l) for l in lists)
    nslot = sum(len((x | y | z) - {last}) for x, y, z in zip(*lists))
    n_dense = sum(r['kind'] > 1 or last in (x | y) for r, x, y in zip(rx, *lists[:2]))
    nnet = sum(sum(r['reactants'].get(s, 0) != r['products'].get(s, 0) for s in x | y) for r, x, y in zip(rx, *lists[:2]))
    doubles = 20 * ns + 4 * nr + 7 * n_fall + ntb + nnet + 1 + 64
    doubles = even(even(doubles) + 128)
    ints = 5 * nr + 6 * (nr + 1) + nreac + nprod + nnet + ntb + nslot + ns
    blob = 8 * doubles + 4 * ((ints + 3) // 4 * 4)
    rhs = 16 + 8 * even(ns) + even(nr)
    jac = rhs + 7 * even(ns) + 3 * even(nr) + 2 * even(n_dense) + even(nslot)
    return blob + 8 * rhs, blob + 8 * jac
