"""Algorithmic work of the path stage, the numerator of the roofline.

The unit is one (path, energy) pair.  Its algorithmic FLOP count is the one tabulated for the reference's literal
port of FEFF's GENFMT (``src/feffgpu/genfmt.py:306-447``: scattering matrices, chain product, termination, trace,
cfac; complex multiply 6, complex add 2, complex x real 2, masked terms excluded), K edge, at a uniform number of
partial waves L = lmax + 1:

    legs          2       3       4       5       6       7       8
    L = 25   12,342  17,246  28,718  40,190  51,662  63,134  74,606
    L = 21   10,534  14,614  24,366  34,118  43,870  53,622  63,374

For every leg count the count is affine in L (the partial-wave sums are linear in L), so the two rows fix it:
flops(nleg, L) = A(nleg) + B(nleg) L.  A path's L at one energy is the mean over its scatterers of
lmax(e, ipot) + 1, the partial-wave limit FEFF applies per scatterer and energy.

This counts what the reference computes, not what this package's kernels execute: they fold the Legendre factors
into the per-path rotation tables, accumulate only the flip-canonical scattering-matrix entries and stream the
spherical-wave recursion, so they issue fewer operations for the same result.
"""
from __future__ import annotations

import numpy as np

_L25 = {2: 12342, 3: 17246, 4: 28718, 5: 40190, 6: 51662, 7: 63134, 8: 74606}
_L21 = {2: 10534, 3: 14614, 4: 24366, 5: 34118, 6: 43870, 7: 53622, 8: 63374}
SLOPE = {n: (_L25[n] - _L21[n]) / 4.0 for n in _L25}
OFFSET = {n: _L25[n] - 25 * SLOPE[n] for n in _L25}
# nine legs continue the per-leg increments
SLOPE[9] = 2 * SLOPE[8] - SLOPE[7]
OFFSET[9] = 2 * OFFSET[8] - OFFSET[7]


def flops_per_energy(nleg: int, L: float) -> float:
    """Algorithmic FLOPs of one path at one energy with (mean) partial-wave count L."""
    return OFFSET[nleg] + SLOPE[nleg] * L


def path_flops(nleg, ipots, lmax_e_ip) -> np.ndarray:
    """Algorithmic FLOPs of every path over all energies (n,): the per-path cost the multi-GPU split balances."""
    nleg = np.asarray(nleg, int)
    ipots = np.asarray(ipots, int)
    L = np.asarray(lmax_e_ip, float) + 1.0
    out = np.zeros(len(nleg))
    for n in np.unique(nleg):
        sel = np.nonzero(nleg == n)[0]
        sc = ipots[sel, 1:n]
        counts = np.zeros((len(sc), L.shape[1]))
        np.add.at(counts, (np.repeat(np.arange(len(sc)), n - 1), sc.ravel()), 1.0)
        mean_L = counts @ L.T / (n - 1)
        out[sel] = np.sum(OFFSET[int(n)] + SLOPE[int(n)] * mean_L, axis=1)
    return out


def batch_flops(nleg, ipots, lmax_e_ip) -> float:
    """Total algorithmic FLOPs of a batch over all energies.  nleg (n,), ipots (n, nleg_max) absorber first,
    lmax_e_ip (E, nph+1) the stage's lmax table."""
    nleg = np.asarray(nleg, int)
    ipots = np.asarray(ipots, int)
    L = np.asarray(lmax_e_ip, float) + 1.0                      # (E, nph+1)
    total = 0.0
    for n in np.unique(nleg):
        sel = nleg == n
        sc = ipots[sel, 1:n]                                    # scatterers' potentials
        # sum over paths and energies of the mean scatterer L: per energy, average L[e, ip] over the scatterers
        counts = np.zeros((len(sc), L.shape[1]))
        np.add.at(counts, (np.repeat(np.arange(len(sc)), n - 1), sc.ravel()), 1.0)
        mean_L = counts @ L.T / (n - 1)                         # (paths, E)
        total += float(np.sum(OFFSET[int(n)] + SLOPE[int(n)] * mean_L))
    return total


# Operations of the form with shared scattering matrices (csrc/fg_shared.cuh), which forms a matrix once per different
# scatterer and energy.  Per partial wave: 20 canonical entries complex x real + add (4), 6 spherical-wave products and 2
# with the t-matrix (6 each), and 5 columns of the recursion (an add and a complex multiply-subtract: 10).  A path of three
# and more legs multiplies its matrices in two blocks, 4 x 4 and 2 x 2, by columns of the final state's entries (four at
# the K edge, six at L and M edges): the first matrix is copied, every further one costs 20 complex multiply-adds (8) a
# column, the last one only the rows that the termination reads (14 at the K edge, all at the others); an Euler phase turns
# two pairs of entries a column (12 each), after the last matrix one at the K edge.  Per path and energy: the termination
# and cfac, about 700.
_SHARED_WAVE = 20 * 4 + 8 * 6 + 5 * 10
_SHARED_END = 700


def _chain_ops(nleg: int, k_edge: bool) -> int:
    """Operations of one path's chain product at one energy."""
    if nleg == 2:
        return 0
    cols, last_rows, last_turns = (4, 14, 1) if k_edge else (6, 20, 2)
    first, middle = cols * 2 * 12, cols * (20 * 8 + 2 * 12)
    return first + (nleg - 3) * middle + cols * (last_rows * 8 + last_turns * 12)


def _legs(x):
    """Leg lengths and the cosines at every atom of paths x (B, nleg, 3), legs 1..nleg (the class of a scatterer up to
    rounding)."""
    import torch
    v = torch.cat([x[:, 1:], x[:, :1]], 1) - x
    r = v.norm(dim=2)
    u = v / r[:, :, None]
    return r, (u * torch.roll(u, -1, 1)).sum(2)


def shared_flops(coords, nleg, ipots, lmax_e_ip, geometry=None, k_edge: bool = True) -> tuple[float, int]:
    """(operations, different scatterers) of a batch whose equal scatterers are formed once: coords (n, nleg_max, 3) A on
    any device.  Scatterers are equal where their two legs, the angle between them and the potential are; geometry maps
    paths (B, nleg, 3) in bohr to (ri, beta, ...) of legs 1..nleg, as GPUPathStage.geometry (the bits that the library
    compares; default: the same quantities by torch)."""
    import torch
    from .pad import BOHR
    c = torch.as_tensor(coords)
    nl = torch.as_tensor(nleg, device=c.device).long()
    ip = torch.as_tensor(ipots, device=c.device).double()
    L = torch.as_tensor(np.asarray(lmax_e_ip, float) + 1.0).sum(0)              # (nph + 1) partial waves over all energies
    E = len(lmax_e_ip)
    keys, total = [], 0.0
    for n in sorted(set(nl.tolist())):
        sel = nl == n
        total += int(sel.sum()) * E * (_SHARED_END + _chain_ops(n, k_edge))
        if n == 2:
            continue
        ri, beta = (geometry or _legs)((c[sel, :n].double() / BOHR).contiguous())[:2]
        for k in range(1, n):                                                   # legs k - 1 -> k and k -> k + 1
            keys.append(torch.stack([ri[:, k - 1], ri[:, k], beta[:, k - 1], ip[sel, k]], 1))
    classes = 0
    if keys:
        u = torch.unique(torch.cat(keys), dim=0)
        classes = int(u.shape[0])
        total += float(L[u[:, 3].long().cpu()].sum()) * _SHARED_WAVE
    two = ip[nl == 2][:, 1].long().cpu()
    return total + float(L[two].sum()) * _SHARED_WAVE, classes
