"""Performance cases: what a user of the Band engine has it do.

Six kinds of work, each through an entry point that a program calls:

* ``bloch``     H(k), S(k) of a resident bundle (``BlochDevice.apply``);
* ``shifted``   factor a batch of shifted pencils H - z S and solve a block of
  right-hand sides with FP64 refinement, for the shifts and (``adjoint``) for
  their conjugates with the same factors (``aosb_factor``, ``aosb_solve``);
* ``subspace``  the FP64 block products of the projected eigenproblem
  (``aosb_spmm_blocks``, ``aosb_gram``, ``aosb_dense_mul``,
  ``aosb_column_norms``);
* ``band``      eigenvalues of an energy window at k points
  (``BandEngine.solve_kpoints``), the whole call;
* ``gamma``     inertia of the real pencil at a new shift
  (``GammaShiftFactor.update_numeric``);
* ``dropin``    shifted solves on host CSR matrices
  (``NativeB200ShiftSolver.solve_shifted``).

Sizes are those of the synthetic workloads and serving stream in
``aospectrum_b200.synth`` (13 or 5 orbitals per atom, periodic sheets and
cubes).  The synthetic generator makes the bundles; matrices H(k), S(k) that a
case takes as given are summed here in 64 bits and rounded to complex64.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from aospectrum_b200 import native, synth
from aospectrum_b200.ciss import CissSettings, EngineSettings, contour_geometry
from aospectrum_b200.data import EnergyInterval, LocalizedOperatorBlocks, LocalizedOperatorBundle
from aospectrum_b200.engine import (BandEngine, BlochDevice, CsrPattern, SymbolicPlan, choose_tile,
                                    row_blocks)
from aospectrum_b200.gamma import GammaShiftFactor
from aospectrum_b200.solvers import NativeB200ShiftSolver
from aospectrum_b200.sparse import SparsePair

CENTRE_EV = -2.57            # middle of the synthetic spectra
STATES_PER_EV = 0.06         # density of states per orbital there


def listed():
    return [
        # one k point of the 64-atom sheet: the smallest call, all latency
        {"name": "bloch_sheet64_1k", "kind": "bloch", "lattice": "sheet", "side": 8,
         "orbitals": 13, "complex": False, "n_k": 1},
        # a step of k points of the 4096-atom cube: the largest Bloch sum
        {"name": "bloch_cube4096_4k", "kind": "bloch", "lattice": "cube", "side": 16,
         "orbitals": 13, "complex": False, "n_k": 4},
        # a contour's node pairs on the 64-atom sheet: few tiles, latency
        {"name": "shifted_sheet64", "kind": "shifted", "lattice": "sheet", "side": 8,
         "orbitals": 13, "pencils": 16, "rhs": 32, "precision": "mixed", "adjoint": True,
         "sweeps": 3},
        # a serving request's small cube with an odd right-hand-side count
        {"name": "shifted_cube343_odd", "kind": "shifted", "lattice": "cube", "side": 7,
         "orbitals": 5, "pencils": 5, "rhs": 17, "precision": "mixed", "adjoint": True,
         "sweeps": 3},
        # part of a k point's node pairs on the 1000-atom cube: the main path
        {"name": "shifted_cube1000", "kind": "shifted", "lattice": "cube", "side": 10,
         "orbitals": 13, "pencils": 8, "rhs": 32, "precision": "mixed", "adjoint": True,
         "sweeps": 4},
        # complex64 factors (one per node, no pairing), 64-wide tiles
        {"name": "plain_cube343", "kind": "shifted", "lattice": "cube", "side": 7,
         "orbitals": 5, "pencils": 8, "rhs": 32, "precision": "plain", "adjoint": False,
         "sweeps": 2},
        # projected problem of a small serving request, ragged widths
        {"name": "subspace_cube343", "kind": "subspace", "lattice": "cube", "side": 7,
         "orbitals": 5, "columns": 96, "kept": 53},
        # projected problem of one k point of the 1000-atom cube (32 x 4 moments)
        {"name": "subspace_cube1000", "kind": "subspace", "lattice": "cube", "side": 10,
         "orbitals": 13, "columns": 128, "kept": 104},
        # one k point, whole call, 64-atom sheet
        {"name": "band_sheet64_1k", "kind": "band", "lattice": "sheet", "side": 8, "orbitals": 13,
         "n_k": 1, "points": 32, "block": 32, "moments": 4, "states": 40, "precision": "mixed"},
        # two k points in one batch, whole call, 1000-atom cube
        {"name": "band_cube1000_2k", "kind": "band", "lattice": "cube", "side": 10,
         "orbitals": 13, "n_k": 2, "points": 32, "block": 32, "moments": 4, "states": 60,
         "precision": "mixed"},
        # one step of a state-counting bisection at Gamma
        {"name": "gamma_cube343", "kind": "gamma", "lattice": "cube", "side": 7, "orbitals": 13},
        # a contour batch on host matrices, through the drop-in solver object
        {"name": "dropin_sheet64", "kind": "dropin", "lattice": "sheet", "side": 8,
         "orbitals": 13, "pencils": 4, "rhs": 32},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["bloch", "shifted", "shifted", "subspace", "band", "gamma", "dropin"])
    lattice = rng.choice(["sheet", "cube"])
    orbitals = rng.choice([5, 13])
    top = {"bloch": 12, "shifted": 8, "subspace": 9, "band": 7, "gamma": 7, "dropin": 5}[kind]
    side = rng.randint(6, 16) if lattice == "sheet" else rng.randint(5, top)
    if kind == "dropin" and lattice == "sheet":
        side = rng.randint(5, 9)
    case = {"kind": kind, "lattice": lattice, "side": side, "orbitals": orbitals}
    n = orbitals * side ** (2 if lattice == "sheet" else 3)
    if kind == "bloch":
        case |= {"complex": rng.random() < 0.3, "n_k": rng.randint(1, 7)}
    elif kind == "shifted":
        precision = rng.choice(["mixed", "mixed", "plain"])
        case |= {"pencils": rng.randint(1, 16 if n < 5000 else 8), "rhs": _log_int(rng, 4, 64),
                 "precision": precision, "adjoint": rng.random() < 0.7,
                 "sweeps": 3 if n < 5000 else 4}
    elif kind == "subspace":
        columns = _log_int(rng, 24, 192)
        case |= {"columns": columns, "kept": rng.randint(columns // 3, columns)}
    elif kind == "band":
        case |= {"n_k": rng.randint(1, 3), "points": rng.choice([16, 24, 32]),
                 "block": rng.choice([16, 24, 32]) if n > 400 else 8,
                 "moments": rng.choice([3, 4]), "states": rng.randint(8, 24) if n > 400 else 6,
                 "precision": rng.choice(["mixed", "mixed", "plain"]) if n < 2000 else "mixed"}
    elif kind == "dropin":
        case |= {"pencils": rng.randint(1, 8), "rhs": _log_int(rng, 4, 48)}
    return case


# ------------------------------------------------------------------- inputs
def _spec(case):
    side = case["side"]
    if case["lattice"] == "sheet":
        return synth.SyntheticSpec(
            name=f"sheet{side}", grid=(side, side, 1), spacing=(2.5, 2.5, 1.0),
            cell=(2.5 * side, 2.5 * side, 15.0), periodic=(True, True, False), cutoff=6.0,
            orbitals_per_atom=case["orbitals"], origin=(0.0, 0.0, 7.5))
    return synth.SyntheticSpec(
        name=f"cube{side}", grid=(side,) * 3, spacing=(2.4,) * 3, cell=(2.4 * side,) * 3,
        periodic=(True,) * 3, cutoff=7.0, orbitals_per_atom=case["orbitals"])


def _bundle(case, seed):
    """The case's structure (atoms, orbitals and block table, the same for
    every seed) with the seed's block values: H scaled by a factor per orbital
    on both sides, S by factors closer to one."""
    bundle = synth.generate_bundle(_spec(case))
    ops, no = bundle.operators, case["orbitals"]
    rng = np.random.default_rng(seed)
    values = []
    for old, spread in ((ops.h_values, 0.1), (ops.s_values, 0.02)):
        u = rng.uniform(1 - spread, 1 + spread, (bundle.basis.n_atoms, no)).astype(np.float32)
        values.append((old.reshape(-1, no, no) * (u[ops.row_atom][:, :, None]
                                                  * u[ops.col_atom][:, None, :])).reshape(-1))
    if case.get("complex"):
        # spin-orbit-like: a unit phase per block, the mirror block carrying
        # the conjugate one, onsite blocks left real
        key = ops.row_atom.astype(np.int64) * bundle.basis.n_atoms + ops.col_atom
        flip = ops.col_atom.astype(np.int64) * bundle.basis.n_atoms + ops.row_atom
        angle = np.sin(1e-3 * (key % 8191)) - np.sin(1e-3 * (flip % 8191))
        phase = np.repeat(np.exp(1j * angle), np.diff(ops.block_offsets))
        values = [(v * phase).astype(np.complex64) for v in values]
    blocks = LocalizedOperatorBlocks(ops.row_atom, ops.col_atom, ops.lattice_shift,
                                     ops.block_offsets, ops.block_shapes, *values)
    return LocalizedOperatorBundle(bundle.structure, bundle.basis, blocks, bundle.filling,
                                   bundle.provenance)


def _kpoints(n_k, seed):
    return np.random.default_rng(seed + 77).uniform(-0.5, 0.5, size=(n_k, 3))


def _plain_bloch(bundle, kpoints):
    """CSR (indptr, indices) and 64-bit H(k), S(k) values [n_k, nnz] of a
    bundle whose atoms all carry the same number of orbitals."""
    ops, atoms = bundle.operators, bundle.basis.n_atoms
    no = bundle.n_orbitals // atoms
    dev = torch.device("cuda")
    pair = torch.from_numpy(ops.row_atom.astype(np.int64) * atoms + ops.col_atom).to(dev)
    groups, member = torch.unique(pair, return_inverse=True)
    gi, gj = groups // atoms, groups % atoms
    mirror = torch.searchsorted(groups, gj * atoms + gi)
    per_row = torch.bincount(gi, minlength=atoms)
    first = torch.cumsum(per_row, 0) - per_row
    rank = torch.arange(groups.numel(), device=dev) - first[gi]
    a = torch.arange(no, device=dev)
    at = ((no * no * first[gi] + no * rank)[:, None, None] + (no * per_row[gi])[:, None, None]
          * a[None, :, None] + a[None, None, :])
    nnz = groups.numel() * no * no
    indices = torch.empty(nnz, dtype=torch.int32, device=dev)
    indices[at.reshape(-1)] = ((no * gj)[:, None, None] + a[None, None, :]).expand(
        at.shape).reshape(-1).to(torch.int32)
    row_len = torch.repeat_interleave(no * per_row, no)
    indptr = torch.zeros(bundle.n_orbitals + 1, dtype=torch.int64, device=dev)
    indptr[1:] = torch.cumsum(row_len, 0)
    shift = torch.from_numpy(ops.lattice_shift.astype(np.float64)).to(dev)
    out = []
    for values in (ops.h_values, ops.s_values):
        v = torch.from_numpy(np.asarray(values)).to(dev).reshape(-1, no, no).to(torch.complex128)
        rows = torch.empty((len(kpoints), nnz), dtype=torch.complex128, device=dev)
        for q, k in enumerate(kpoints):
            turn = shift @ torch.as_tensor(k, dtype=torch.float64, device=dev)
            phase = torch.polar(torch.ones_like(turn), 2.0 * math.pi * turn)
            x = torch.zeros((groups.numel(), no, no), dtype=torch.complex128, device=dev)
            x.index_add_(0, member, v * phase[:, None, None])
            x = 0.5 * (x + x[mirror].mH)
            rows[q, at.reshape(-1)] = x.reshape(-1)
        out.append(rows)
    return indptr, indices, out[0], out[1]


def _matrices(case, seed, k=None):
    """Bundle, CSR pattern (host) and complex64 H, S values (device, [nnz])."""
    bundle = _bundle(case, seed)
    indptr, indices, h, s = _plain_bloch(bundle, _kpoints(1, seed) if k is None else [k])
    return (bundle, indptr.cpu().numpy(), indices.cpu().numpy(), h[0].to(torch.complex64),
            s[0].to(torch.complex64))


def _shifts(case, n):
    """Upper-half contour nodes around a window of up to 200 states with the
    0.02 eV guards of a band calculation."""
    half = 0.02 + 0.5 * min(200, n // 20) / (STATES_PER_EV * n)
    z, _, _ = contour_geometry(EnergyInterval(CENTRE_EV - half, CENTRE_EV + half),
                               CissSettings(integration_points=2 * case["pencils"]))
    return z[:case["pencils"]].astype(np.complex128)


def _random(shape, seed, dtype=torch.complex128):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, dtype=dtype, device="cuda", generator=g)


def _sizes(case):
    n = case["orbitals"] * case["side"] ** (2 if case["lattice"] == "sheet" else 3)
    return n, n // case["orbitals"]


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    return {"kind": case["kind"], **_PREPARE[case["kind"]](case, seed)}


def _prepare_bloch(case, seed):
    bundle = _bundle(case, seed)
    return {"bloch": BlochDevice(bundle, torch.device("cuda", 0)),
            "k": _kpoints(case["n_k"], seed)}


def _prepare_shifted(case, seed):
    dev = torch.device("cuda", 0)
    bundle, indptr, indices, h, s = _matrices(case, seed)
    n, P, L = bundle.n_orbitals, case["pencils"], case["rhs"]
    mixed = case["precision"] == "mixed"
    atoms = np.asarray(bundle.basis.atom_offsets)
    pattern = CsrPattern(n, indptr, indices, dev)
    plan = SymbolicPlan(n, indptr, indices, tile=128 if mixed else choose_tile(n),
                        supervariables=atoms, device=dev)
    blocks = row_blocks(indptr, indices, starts=atoms[:-1])
    lib = native.library()
    precision = native.PRECISION_BF16X3 if mixed else native.PRECISION_PLAIN

    def raw(count):
        return torch.empty(max(int(count), 16), dtype=torch.uint8, device=dev)

    z = torch.from_numpy(_shifts(case, n)).to(dev)
    state = {
        "n": n, "P": P, "L": L, "nnz": pattern.nnz, "precision": precision, "plan": plan,
        "pattern": pattern, "h": h, "s": s, "z": z, "zc": torch.conj_physical(z),
        "flags": native.SOLVE_TENSOR_CORES if mixed else 0, "sweeps": case["sweeps"],
        "directions": 2 if case["adjoint"] else 1,
        "blocks": torch.from_numpy(blocks).to(dev), "max_rows": int(np.diff(blocks).max()),
        "pk": torch.zeros(P, dtype=torch.int32, device=dev),
        "factor": raw(lib.aosb_factor_bytes(plan.handle, P)),
        "pivots": torch.empty((P, plan.info.n_pad), dtype=torch.int32, device=dev),
        "status": torch.zeros(P, dtype=torch.int32, device=dev),
        "workspace": raw(lib.aosb_factor_workspace_bytes(plan.handle, P, precision)),
        "scratch": raw(lib.aosb_solve_scratch_bytes(plan.handle, P, L)),
        "work": torch.empty((P, plan.info.n_pad, L), dtype=torch.complex64, device=dev),
        "b": _random((P, n, L), seed),
        "r": torch.empty((P, n, L), dtype=torch.complex128, device=dev),
    }
    state["x"] = [torch.empty_like(state["r"]) for _ in range(state["directions"])]
    return state


def _prepare_subspace(case, seed):
    dev = torch.device("cuda", 0)
    bundle, indptr, indices, h, s = _matrices(case, seed)
    n, p, r = bundle.n_orbitals, case["columns"], case["kept"]
    pattern = CsrPattern(n, indptr, indices, dev)
    blocks = row_blocks(indptr, indices, starts=np.asarray(bundle.basis.atom_offsets)[:-1])
    scratch = native.library().aosb_gram_scratch_bytes(n, p, p)
    moments, transform, energies = _subspace_inputs(n, p, r, seed)
    return {
        "n": n, "pattern": pattern, "h": h, "s": s, "moments": moments, "transform": transform,
        "energies": energies, "blocks": torch.from_numpy(blocks).to(dev),
        "max_rows": int(np.diff(blocks).max()),
        "scratch": torch.empty(max(int(scratch), 16), dtype=torch.uint8, device=dev),
    }


def _subspace_inputs(n, p, r, seed):
    return (_random((n, p), seed + 1) / math.sqrt(n), _random((p, r), seed + 2) / math.sqrt(p),
            CENTRE_EV + 0.1 * _random((r,), seed + 3, torch.float64))


def _settings(case):
    return CissSettings(integration_points=case["points"], block_size=case["block"],
                        moment_size=case["moments"])


def _window(case):
    half = 0.5 * case["states"] / (STATES_PER_EV * _sizes(case)[0])
    return EnergyInterval(CENTRE_EV - half, CENTRE_EV + half)


def _prepare_band(case, seed):
    engine = BandEngine(_bundle(case, seed), _settings(case),
                        EngineSettings(precision=case["precision"]))
    return {"engine": engine, "k": _kpoints(case["n_k"], seed).tolist(), "window": _window(case),
            "most": engine.settings.search_dimension}


def _gamma_shift(seed):
    return float(CENTRE_EV + np.random.default_rng(seed + 5).uniform(-1.0, 1.0))


def _prepare_gamma(case, seed):
    bundle, indptr, indices, h, s = _matrices(case, seed, (0.0, 0.0, 0.0))
    factor = GammaShiftFactor(bundle.n_orbitals, indptr, indices, h.real.contiguous(),
                              s.real.contiguous(), CENTRE_EV)
    return {"factor": factor, "shift": _gamma_shift(seed)}


def _prepare_dropin(case, seed):
    from scipy import sparse

    bundle, indptr, indices, h, s = _matrices(case, seed)
    n = bundle.n_orbitals
    ip = indptr.astype(np.int32)
    pair = SparsePair(*(sparse.csr_matrix((v.cpu().numpy(), indices, ip), shape=(n, n), copy=False)
                        for v in (h, s)), (0.0, 0.0, 0.0))
    rhs = _random((n, case["rhs"]), seed).to(torch.complex64).cpu().numpy()
    return {"solver": NativeB200ShiftSolver(), "pair": pair, "rhs": rhs,
            "z": _shifts(case, n).astype(np.complex64)}


_PREPARE = {"bloch": _prepare_bloch, "shifted": _prepare_shifted, "subspace": _prepare_subspace,
            "band": _prepare_band, "gamma": _prepare_gamma, "dropin": _prepare_dropin}


# ---------------------------------------------------------------------- run
def run(state):
    return _RUN[state["kind"]](state)


def _run_bloch(t):
    return list(t["bloch"].apply(t["k"]))


def _run_shifted(t):
    C, plan, n, P, L = native.C, t["plan"].handle, t["n"], t["P"], t["L"]
    stream = torch.cuda.current_stream().cuda_stream
    t["status"].zero_()
    fa = native.FactorArgs(native.ABI_VERSION, C.sizeof(native.FactorArgs), P, t["precision"],
                           t["h"].data_ptr(), t["s"].data_ptr(), t["pk"].data_ptr(),
                           t["z"].data_ptr(), t["factor"].data_ptr(), t["pivots"].data_ptr(),
                           t["status"].data_ptr(), t["workspace"].data_ptr(), stream)
    native.call("aosb_factor", plan, C.byref(fa))
    for adjoint in range(t["directions"]):
        x, z = t["x"][adjoint], t["zc"] if adjoint else t["z"]
        sa = native.SolveArgs(native.ABI_VERSION, C.sizeof(native.SolveArgs), P, L, adjoint,
                              t["flags"], t["factor"].data_ptr(), t["pivots"].data_ptr(),
                              t["work"].data_ptr(), t["scratch"].data_ptr(), stream)
        for sweep in range(t["sweeps"] + 1):
            src = t["r"] if sweep else t["b"]
            native.call("aosb_gather_rhs", plan, P, L, src.data_ptr(), n * L,
                        t["work"].data_ptr(), stream)
            native.call("aosb_solve", plan, C.byref(sa))
            native.call("aosb_scatter_solution", plan, P, L, t["work"].data_ptr(), x.data_ptr(),
                        1 if sweep else 0, stream)
            if sweep < t["sweeps"]:
                native.call("aosb_shifted_residual_blocks", n, L, P, t["blocks"].numel() - 1,
                            t["blocks"].data_ptr(), t["max_rows"], t["pattern"].d_indptr,
                            t["pattern"].d_indices, t["h"].data_ptr(), t["s"].data_ptr(),
                            t["nnz"], t["pk"].data_ptr(), z.data_ptr(), t["b"].data_ptr(), n * L,
                            x.data_ptr(), t["r"].data_ptr(), stream)
        native.call("aosb_solve_check", plan, C.byref(sa))
    return t["x"] + [t["status"]]


def _run_subspace(t):
    n, pattern, stream = t["n"], t["pattern"], torch.cuda.current_stream().cuda_stream

    def product(values, x):
        y = torch.empty_like(x)
        native.call("aosb_spmm_blocks", n, x.shape[1], t["blocks"].numel() - 1,
                    t["blocks"].data_ptr(), t["max_rows"], pattern.d_indptr, pattern.d_indices,
                    values.data_ptr(), pattern.nnz, x.data_ptr(), x.stride(0), y.data_ptr(),
                    y.stride(0), stream)
        return y

    def gram(x, y):
        g = torch.empty((x.shape[1], y.shape[1]), dtype=torch.complex128, device=x.device)
        native.call("aosb_gram", n, x.shape[1], y.shape[1], x.data_ptr(), x.stride(0),
                    y.data_ptr(), y.stride(0), g.data_ptr(), t["scratch"].data_ptr(), stream)
        return g

    moments, transform = t["moments"], t["transform"]
    overlap = gram(moments, product(t["s"], moments))
    p, r = transform.shape
    basis = torch.empty((n, r), dtype=torch.complex128, device=moments.device)
    native.call("aosb_dense_mul", n, p, r, moments.data_ptr(), moments.stride(0),
                transform.data_ptr(), basis.data_ptr(), basis.stride(0), stream)
    hb, sb = product(t["h"], basis), product(t["s"], basis)
    norms = torch.empty(r, dtype=torch.float64, device=moments.device)
    native.call("aosb_column_norms", n, r, hb.data_ptr(), sb.data_ptr(), hb.stride(0),
                t["energies"].data_ptr(), norms.data_ptr(), stream)
    return [overlap, basis, gram(basis, hb), gram(basis, sb), norms]


def _run_band(t):
    results, _ = t["engine"].solve_kpoints(t["k"], t["window"])
    return [_row(r.energies_ev, t["most"]) for r in results]


def _row(energies, most):
    """A k point's energies in a row of a table as wide as the search space."""
    row = np.zeros(most, dtype=energies.dtype)
    row[:energies.size] = energies
    return row


def _run_gamma(t):
    at = t["factor"].update_numeric(t["shift"]).inertia
    return [at.below, at.zero, at.above]


def _run_dropin(t):
    return [t["solver"].solve_shifted(t["pair"], t["z"], t["rhs"]).solutions]


_RUN = {"bloch": _run_bloch, "shifted": _run_shifted, "subspace": _run_subspace,
        "band": _run_band, "gamma": _run_gamma, "dropin": _run_dropin}


# --------------------------------------------------------------------- work
def work(case):
    """Bytes: inputs read once and outputs written once.  Flops: eight real
    operations per complex product and sum (two in a real one)."""
    kind, (n, atoms), no = case["kind"], _sizes(case), case["orbitals"]
    bundle = synth.generate_bundle(_spec(case))
    ops = bundle.operators
    nnz = no * no * np.unique(ops.row_atom.astype(np.int64) * atoms + ops.col_atom).size
    values = int(ops.block_offsets[-1])
    if kind == "bloch":
        item = 8 if case["complex"] else 4
        return {"bytes": 2 * values * item + 16 * nnz * case["n_k"],
                "flops": 8 * values * case["n_k"]}
    if kind == "subspace":
        p, r = case["columns"], case["kept"]
        return {"bytes": 20 * nnz + 16 * n * (p + r) + 16 * (p * p + p * r + 2 * r * r),
                "flops": 8 * (nnz * (p + 2 * r) + n * (p * p + p * r + 2 * r * r))}
    flops, entries = _elimination(case, bundle)
    if kind == "gamma":
        return {"bytes": 8 * nnz, "flops": flops / 4}
    if kind == "band":
        pencils, L, steps = case["n_k"] * case["points"] / 2, case["block"], 1
        if case["precision"] == "plain":
            pencils, steps = 2 * pencils, 0
        solves = case["n_k"] * case["points"]
        p = L * case["moments"]
        each = (steps + 1) * 8 * entries * L + steps * 8 * nnz * L
        return {"bytes": 8 * values + 8 * n * L,
                "flops": pencils * flops + solves * each
                + case["n_k"] * 8 * (3 * nnz * p + 3 * n * p * p)}
    P, L = case["pencils"], case["rhs"]
    if kind == "dropin":
        return {"bytes": 16 * nnz + 8 * n * L * (1 + P),
                "flops": P * (flops + 3 * 8 * entries * L + 2 * 8 * nnz * L)}
    both, sweeps = 2 if case["adjoint"] else 1, case["sweeps"]
    return {"bytes": 20 * nnz + 16 * P * n * L * (1 + both),
            "flops": P * (flops + both * ((sweeps + 1) * 8 * entries * L
                                          + sweeps * 8 * nnz * L))}


def _elimination(case, bundle):
    """Flops of one complex elimination and entries of its factors, from the
    symbolic analysis (padding excluded from the flops)."""
    dev = torch.device("cuda", 0)
    bloch = BlochDevice(bundle, dev, upload=False)
    plan = SymbolicPlan(bloch.n, bloch.indptr, bloch.indices, tile=64,
                        supervariables=np.asarray(bundle.basis.atom_offsets), device=dev,
                        upload=False)
    found = plan.info.factor_flops_alg, plan.info.n_slots * plan.info.tile ** 2
    plan.close()
    bloch.close()
    return found


# -------------------------------------------------------------------- exact
def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def _exact_bloch(case, seed):
    _, _, h, s = _plain_bloch(_bundle(case, seed), _kpoints(case["n_k"], seed))
    return [h, s]


def _dense(indptr, indices, values, n):
    ip = torch.from_numpy(indptr).to(values.device)
    rows = torch.repeat_interleave(torch.arange(n, device=values.device), ip[1:] - ip[:-1])
    out = torch.zeros((n, n), dtype=torch.complex128, device=values.device)
    out[rows, torch.from_numpy(indices).to(values.device).long()] = values.to(torch.complex128)
    return out


def _exact_shifted(case, seed):
    _, indptr, indices, h, s = _matrices(case, seed)
    n, P, L = indptr.size - 1, case["pencils"], case["rhs"]
    b = _random((P, n, L), seed)
    directions = 2 if case["adjoint"] else 1
    out = [torch.empty_like(b) for _ in range(directions)]
    hd, sd = _dense(indptr, indices, h, n), _dense(indptr, indices, s, n)
    for p, z in enumerate(_shifts(case, n)):
        lu, piv = torch.linalg.lu_factor(hd - complex(z) * sd)
        for d in range(directions):
            out[d][p] = torch.linalg.lu_solve(lu, piv, b[p], adjoint=bool(d))
    return out + [None]


def _exact_subspace(case, seed):
    _, indptr, indices, h, s = _matrices(case, seed)
    n = indptr.size - 1
    m, t, e = _subspace_inputs(n, case["columns"], case["kept"], seed)
    hd, sd = _dense(indptr, indices, h, n), _dense(indptr, indices, s, n)
    basis = m @ t
    hb, sb = hd @ basis, sd @ basis
    return [m.mH @ (sd @ m), basis, basis.mH @ hb, basis.mH @ sb,
            torch.linalg.vector_norm(hb - e * sb, dim=0)]


def _exact_band(case, seed):
    if _sizes(case)[0] > 3000:
        return None
    bundle, window = _bundle(case, seed), _window(case)
    indptr, indices, h, s = _plain_bloch(bundle, _kpoints(case["n_k"], seed))
    indptr, indices, n = indptr.cpu().numpy(), indices.cpu().numpy(), bundle.n_orbitals
    out = []
    for q in range(case["n_k"]):
        hd, sd = _dense(indptr, indices, h[q], n), _dense(indptr, indices, s[q], n)
        low = torch.linalg.cholesky(sd)
        a = torch.linalg.solve_triangular(low, hd, upper=False)
        a = torch.linalg.solve_triangular(low, a.mH, upper=False)
        e = torch.linalg.eigvalsh(0.5 * (a + a.mH))
        e = e[(e > window.lower_ev) & (e < window.upper_ev)].cpu().numpy()
        out.append(_row(e, _settings(case).search_dimension))
    return out


def _exact_dropin(case, seed):
    _, indptr, indices, h, s = _matrices(case, seed)
    n = indptr.size - 1
    b = _random((n, case["rhs"]), seed).to(torch.complex64).to(torch.complex128)
    # the solver object takes H - z S in complex64, as its reference does
    z = torch.from_numpy(_shifts(case, n).astype(np.complex64)).to(h.device)
    hz = [(h.cpu().numpy() - v * s.cpu().numpy()).astype(np.complex64) for v in z.cpu().numpy()]
    return [torch.stack([torch.linalg.solve(
        _dense(indptr, indices, torch.from_numpy(a).to(h.device), n), b) for a in hz]).cpu().numpy()]


_EXACT = {"bloch": _exact_bloch, "shifted": _exact_shifted, "subspace": _exact_subspace,
          "band": _exact_band, "gamma": lambda case, seed: None, "dropin": _exact_dropin}
