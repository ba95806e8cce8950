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
