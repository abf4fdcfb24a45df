"""Timed cases of the engine: the calls a plane-wave program makes, through
the public entry points of `pspw`, over the range of cells it meets.

A case is a dict of plain values; `kind` says which call it is:

  hpsi    block H*psi on device blocks (Cell.apply_ham_block_dev)
  filter  the Chebyshev filter on a device block (Cell.chebyfilt_dev)
  batch   H*psi on several cells in one launch (Batch.apply)
  rho     density and kinetic energy of a block (pspw_eval_rho_psi_dev)
  ortho   orthonormal basis of a block (Cell.ortho_span_dev)
  eig     eigendecomposition of the Rayleigh-Ritz matrix (Cell.eig_zheevd_dev)
  scf     iterations of the whole SCF loop from an INPUT (System.cheby_scf)

Cells are diamond-cubic silicon supercells (`nrep`^3 conventional cells) or
orthorhombic cells of random atoms (`a`, `b`, `c` in bohr, `nat` atoms).
`grid` is the length of a forced cubic grid, 0 for the reference's own grid
rule, or -1 for the smallest 5-smooth length per axis.
"""
import ctypes
import functools
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "ffr-pspw-dft-c_b200"))

from pspw import PREC_F32, PREC_F64, Cell, check, lib, synth  # noqa: E402
from pspw.batch import Batch  # noqa: E402
from pspw.cell import basis_gamma  # noqa: E402
from pspw.inputs import write_input, write_synthetic_fhi  # noqa: E402
from pspw.serve import smooth_grid  # noqa: E402
from pspw.system import System  # noqa: E402

DEV = "cuda:0"
LB, UB = 0.5, 18.0  # filter window (Ha): above the wanted states, up to the spectrum's end
WNL = (1.5, 0.8, 0.8, 0.8)


def listed():
    return [
        # one vector on a small cell: every H*v of the Lanczos filter bounds
        dict(name="hpsi_f64_si8_vector", kind="hpsi", prec=64, nrep=1, grid=32, ecut=15.0, nb=1),
        # a small cell's whole block, as the first steps of a small job apply it
        dict(name="hpsi_f32_si8_block", kind="hpsi", prec=32, nrep=1, grid=32, ecut=15.0, nb=16),
        # a cell whose INPUT forces no grid: the reference's rule (74^3 here), FP64
        dict(name="hpsi_f64_si64_rule", kind="hpsi", prec=64, nrep=2, grid=0, ecut=15.0, nb=32),
        # a molecule-sized orthorhombic cell: three grid lengths, an odd band count
        dict(name="hpsi_f32_ortho", kind="hpsi", prec=32, a=11.3, b=14.9, c=9.7, nat=11,
             atoms_seed=5, grid=-1, ecut=22.0, nb=93),
        # the filter of the mixed-precision SCF loop on Si64, the benchmark's step
        dict(name="filter_f32_si64", kind="filter", prec=32, nrep=2, grid=64, ecut=15.0, nb=144,
             degree=10),
        # the same in the reference's own precision
        dict(name="filter_f64_si64", kind="filter", prec=64, nrep=2, grid=64, ecut=15.0, nb=144,
             degree=10),
        # the largest cell of the benchmark: one application to the 512 states of
        # Si216, as each step of the block eigensolvers makes in FP64
        dict(name="hpsi_f64_si216", kind="hpsi", prec=64, nrep=3, grid=96, ecut=15.0, nb=512),
        # several uneven cells at once, as a screening run applies them
        dict(name="batch_f32_6cells", kind="batch", prec=32, ncells=6, cells_seed=11),
        # the density after each Rayleigh-Ritz step
        dict(name="rho_si64", kind="rho", nrep=2, grid=64, ecut=15.0, nb=142),
        # the orthonormalisation after each filter
        dict(name="ortho_si64", kind="ortho", nrep=2, grid=64, ecut=15.0, nb=146),
        # the Rayleigh-Ritz eigenproblem of the same loop
        dict(name="eig_146", kind="eig", n=146),
        # three iterations of the whole FP64 loop on Si64
        dict(name="scf_f64_si64", kind="scf", nrep=2, grid=64, iters=3, nempty=14),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_cell(rng):
    """A silicon supercell on a forced or rule grid, or an orthorhombic cell."""
    pick = rng.random()
    if pick < 0.25:
        return dict(nrep=1, grid=rng.choice([0, 24, 30, 32, 36]),
                    ecut=round(rng.uniform(8.0, 15.0), 2))
    if pick < 0.5:
        return dict(nrep=2, grid=rng.choice([0, 60, 64, 72]), ecut=round(rng.uniform(10.0, 15.0), 2))
    return dict(a=round(rng.uniform(8.0, 16.0), 2), b=round(rng.uniform(8.0, 16.0), 2),
                c=round(rng.uniform(8.0, 16.0), 2), nat=rng.randint(2, 16),
                atoms_seed=rng.randrange(1000), grid=rng.choice([0, -1, -1]),
                ecut=round(rng.uniform(10.0, 25.0), 2))


def draw(rng):
    kind = rng.choice(["hpsi"] * 5 + ["filter"] * 4 + ["rho", "rho", "batch", "ortho", "eig", "scf"])
    if kind == "eig":
        return dict(kind=kind, n=_logint(rng, 8, 150))
    if kind == "batch":
        return dict(kind=kind, prec=rng.choice([32, 32, 64]), ncells=rng.randint(2, 8),
                    cells_seed=rng.randrange(1000))
    if kind == "scf":
        return dict(kind=kind, nrep=1, grid=rng.choice([0, 32]), iters=rng.randint(2, 4),
                    nempty=rng.randint(2, 9))
    case = dict(kind=kind, nb=_logint(rng, 2 if kind == "ortho" else 1, 256), **_draw_cell(rng))
    if kind == "ortho":
        case["nb"] = min(case["nb"], 150)
    if kind in ("hpsi", "filter"):
        case["prec"] = rng.choice([32, 64])
    if kind == "filter":
        case["degree"] = rng.randint(4, 12)
    return case


# ---------------------------------------------------------------- geometry
def _lattice(case):
    if "nrep" in case:
        return synth.si_diamond(case["nrep"])
    abc = np.array([case["a"], case["b"], case["c"]])
    rng = np.random.default_rng(case["atoms_seed"])
    best = None
    for _ in range(200):  # the most open of some random placements
        p = rng.uniform(0.0, 1.0, (case["nat"], 3)) * abc
        d = p[:, None] - p[None]
        d -= np.round(d / abc) * abc
        r = np.sqrt((d * d).sum(-1)) + 1e9 * np.eye(len(p))
        if best is None or r.min() > best[0]:
            best = (r.min(), p)
    return np.diag(abc), best[1]


@functools.lru_cache(maxsize=8)
def _basis(key):
    """Basis and projectors of a cell in the reference's layouts."""
    case = dict(key)
    lat, pos = _lattice(case)
    grid, ecut = case["grid"], case["ecut"]
    if grid > 0:
        nr = (grid,) * 3
    elif grid == 0:
        nr = None
    else:
        gmax = math.sqrt(8.0 * ecut)
        nr = tuple(smooth_grid(gmax * lat[i, i] / math.pi + 1.0) for i in range(3))
    b = basis_gamma(lat, 2.0 * ecut, nr, [len(pos)], [pos])
    # a projector's norm sum_G |beta|^2 grows with the cell: weights per norm
    norm = b["omega"] * math.pi ** 1.5 / (2.0 * math.pi) ** 3
    pkg_a, wnl = synth.kb_form_factors(b, lat, weights=tuple(w / norm for w in WNL))
    b.update(pkg_a=pkg_a, wnl=wnl, lm_end=[4], lattice=lat, positions=pos)
    return b


def _basis_of(case):
    keep = ("nrep", "a", "b", "c", "nat", "atoms_seed", "grid", "ecut")
    return _basis(tuple((k, case[k]) for k in keep if k in case))


def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _veff(b, g):
    """Gaussian wells at slightly displaced atoms, on the grid (NR1 fastest)."""
    n1, n2, n3 = b["nr"]
    recip = 2.0 * math.pi * np.linalg.inv(b["lattice"]).T
    pos = torch.tensor(b["positions"], device=DEV)
    pos = pos + 0.1 * torch.randn(pos.shape, generator=g, device=DEV, dtype=torch.float64)
    gs = [torch.fft.fftfreq(n, 1.0 / n, device=DEV, dtype=torch.float64) * recip[i, i]
          for i, n in enumerate((n1, n2, n3))]
    ph = [torch.exp(-1j * pos[:, i, None] * gs[i][None]) for i in range(3)]
    yz = (ph[2][:, :, None] * ph[1][:, None, :]).reshape(len(pos), -1)
    w = 1.2
    fs = [torch.exp(-0.5 * w * w * x * x) for x in gs]
    form = -2.0 * (2.0 * math.pi * w * w) ** 1.5 * (
        fs[2][:, None, None] * fs[1][None, :, None] * fs[0][None, None, :])
    v = torch.fft.ifftn((yz.T @ ph[0]).reshape(n3, n2, n1) * form)
    return (v.real * (n1 * n2 * n3 / b["omega"])).reshape(-1).contiguous()


def _block(b, nb, g, orthonormal=True):
    """Wavefunctions, one band per row: random plane-wave coefficients that
    fall off as exp(-|G|^2/2), i.e. low states as a loop holds them after its
    first filter, orthonormalised."""
    ngw = b["ngw"]
    x = torch.randn(nb, ngw, 2, generator=g, device=DEV, dtype=torch.float64)
    x = torch.view_as_complex(x)
    g2 = torch.tensor(np.asarray(b["xkg"][:ngw]) * b["tpiba"] ** 2, device=DEV)
    x = x * torch.exp(-g2 / 2.0)[None]
    if orthonormal:
        x = torch.linalg.qr(x.T)[0].T.contiguous()
    return x


def _cell_inputs(case, seed):
    """What the kernels are given, made from the seed: V_eff and the block."""
    b, g = _basis_of(case), _rng(seed)
    nb = min(case["nb"], b["ngw"])
    veff = _veff(b, g)
    x = _block(b, nb, g)
    if case.get("prec") == 32:
        x = x.to(torch.complex64)
    return b, veff, x, g


def _make_cell(b, veff):
    cell = Cell.from_arrays(b)
    torch.cuda.synchronize()
    check(lib().pspw_cell_set_veff_device(cell.handle, veff.data_ptr(), veff.numel()))
    torch.cuda.synchronize()
    return cell


def _prec(case):
    return PREC_F32 if case["prec"] == 32 else PREC_F64


def _batch_cases(case):
    """Cells of a screening run: 8-16 bohr, 2-16 atoms, 8-256 bands."""
    rng = np.random.default_rng(case["cells_seed"])
    out = []
    for _ in range(case["ncells"]):
        a, b, c = (round(float(v), 2) for v in rng.uniform(8.0, 16.0, 3))
        out.append(dict(a=a, b=b, c=c, nat=int(rng.integers(2, 17)),
                        atoms_seed=int(rng.integers(1000)), grid=-1,
                        ecut=round(float(rng.uniform(10.0, 25.0)), 2),
                        nb=int(rng.integers(8, 257)), prec=case["prec"]))
    return out


def _dense_hermitian(n, seed):
    g = _rng(seed)
    q = torch.randn(n, n, 2, generator=g, device=DEV, dtype=torch.float64)
    q = torch.linalg.qr(torch.view_as_complex(q))[0]
    u = torch.rand(n, generator=g, device=DEV, dtype=torch.float64)
    w = 0.02 * torch.arange(n, device=DEV, dtype=torch.float64) + 0.008 * u - 0.3
    h = (q * w) @ q.conj().T
    return 0.5 * (h + h.conj().T)


class _DeviceBlock:
    """A block the engine owns, for torch.as_tensor; the tensor keeps this
    object and with it the block's owner alive."""

    def __init__(self, owner, ptr, shape, prec):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, data=(ptr, False), version=3,
                                             typestr="<c8" if prec == PREC_F32 else "<c16")


def _system_positions(case, seed):
    lat, pos = synth.si_diamond(case["nrep"])
    return lat, pos + np.random.default_rng(seed).uniform(-0.1, 0.1, pos.shape)


# ---------------------------------------------------------------- the calls
def prepare(case, seed):
    kind = case["kind"]
    if kind == "eig":
        a0 = _dense_hermitian(case["n"], seed).T.contiguous()  # column-major
        b = _basis_of(dict(nrep=1, grid=24, ecut=4.0))
        cell = Cell.from_arrays(b)
        return dict(kind=kind, cell=cell, stream=torch.cuda.ExternalStream(cell.stream()), a0=a0,
                    a=torch.empty_like(a0), n=case["n"],
                    w=torch.zeros(case["n"], device=DEV, dtype=torch.float64))
    if kind == "scf":
        lat, pos = _system_positions(case, seed)
        with tempfile.TemporaryDirectory() as d:
            write_synthetic_fhi(os.path.join(d, "X.fhi"))
            grid = (case["grid"],) * 3 if case["grid"] > 0 else None
            write_input(os.path.join(d, "INPUT"), "X.fhi", pos, float(lat[0][0]), ecut_ry=30.0,
                        idiag=-1, imix=3, max_scf=case["iters"], nempty=case["nempty"],
                        fft_grid=grid, conv=1e-12)
            return dict(kind=kind, system=System(d))
    if kind == "batch":
        subs = _batch_cases(case)
        cells, blocks = [], []
        for i, sub in enumerate(subs):
            b, veff, x, _ = _cell_inputs(sub, seed + 1000 * i)
            cells.append(_make_cell(b, veff))
            blocks.append(x)
        batch = Batch(cells, [len(x) for x in blocks], _prec(case))
        outs = []
        for i, x in enumerate(blocks):
            batch.upload(i, x.cpu().numpy().T)
            d_in, d_out = ctypes.c_void_p(), ctypes.c_void_p()
            check(lib().pspw_batch_blocks(batch._h, i, ctypes.byref(d_in), ctypes.byref(d_out)))
            outs.append(torch.as_tensor(_DeviceBlock(batch, d_out.value, tuple(x.shape),
                                                     _prec(case)),
                                        device=DEV))
        return dict(kind=kind, batch=batch, outs=outs)
    b, veff, x, g = _cell_inputs(case, seed)
    cell = _make_cell(b, veff)
    nb, ngw = x.shape
    state = dict(kind=kind, cell=cell, nb=nb, ngw=ngw, x0=x,
                 stream=torch.cuda.ExternalStream(cell.stream()))
    if kind in ("hpsi", "filter"):
        state.update(prec=_prec(case), out=torch.empty_like(x), degree=case.get("degree"))
    elif kind == "rho":
        # two electrons in each occupied state, the top tenth empty
        state.update(focc=np.where(np.arange(nb) < max(1, (9 * nb) // 10), 2.0, 0.0),
                     omega=b["omega"],
                     rho=torch.zeros(veff.numel(), device=DEV, dtype=torch.float64))
    elif kind == "ortho":
        # what a filter leaves: the wanted states mixed at random
        m = torch.randn(nb, nb, 2, generator=g, device=DEV, dtype=torch.float64)
        state.update(x0=(torch.view_as_complex(m) @ x).contiguous(), out=torch.empty_like(x))
    torch.cuda.synchronize()
    return state


def run(s):
    kind = s["kind"]
    if kind == "hpsi":
        s["cell"].apply_ham_block_dev(s["x0"], s["out"], s["ngw"], s["ngw"], s["nb"], s["prec"])
        return s["out"]
    if kind == "filter":  # in place, on a copy of the block the program keeps
        with torch.cuda.stream(s["stream"]):
            s["out"].copy_(s["x0"])
        s["cell"].chebyfilt_dev(s["out"], s["ngw"], s["ngw"], s["nb"], s["degree"], LB, UB,
                                s["prec"])
        return s["out"]
    if kind == "batch":
        s["batch"].apply()
        return s["outs"]
    if kind == "rho":
        with torch.cuda.stream(s["stream"]):
            s["rho"].zero_()
        ekin = ctypes.c_double(0.0)
        check(lib().pspw_eval_rho_psi_dev(s["cell"].handle, s["rho"].data_ptr(),
                                          s["x0"].data_ptr(), s["ngw"], s["ngw"], s["nb"],
                                          s["focc"].ctypes.data, 1.0, s["omega"],
                                          ctypes.byref(ekin)))
        return dict(rho=s["rho"], ekin=ekin.value)
    if kind == "ortho":
        with torch.cuda.stream(s["stream"]):
            s["out"].copy_(s["x0"])
        s["cell"].ortho_span_dev(s["out"], s["ngw"], s["nb"])
        return s["out"]
    if kind == "eig":
        with torch.cuda.stream(s["stream"]):
            s["a"].copy_(s["a0"])
        s["cell"].eig_zheevd_dev(s["a"], s["n"], s["w"], s["n"])
        return dict(vectors=s["a"], values=s["w"])
    r = s["system"].cheby_scf(PREC_F64)
    return dict(eig=r["eig"], hist=np.ascontiguousarray(r["hist"][:, :3]),
                energies=[float(r["energies"][k]) for k in sorted(r["energies"])])


# ---------------------------------------------------------------- what a pass needs
def _estimate(case):
    """(NGW, NNR, atoms) of a cell without building it."""
    if "nrep" in case:
        abc, nat = [synth.SI_A0 * case["nrep"]] * 3, 8 * case["nrep"] ** 3
    else:
        abc, nat = [case["a"], case["b"], case["c"]], case["nat"]
    ecut = case.get("ecut", 15.0)
    omega = abc[0] * abc[1] * abc[2]
    ngw = omega * (2.0 * ecut) ** 1.5 / (6.0 * math.pi ** 2)
    nnr = 1.0
    for length in abc:
        nnr *= case["grid"] if case["grid"] > 0 else math.sqrt(8.0 * ecut) * length / math.pi + 2
    return ngw, nnr, nat


def _hpsi_work(case, nb, applications=1):
    ngw, nnr, nat = _estimate(case)
    sc = 8 if case.get("prec") == 32 else 16
    data = nb * 2 * ngw * sc + nnr * sc / 2 + ngw * (nat * sc + 4 * sc / 2 + 4 + sc / 2)
    flops = nb * (2 * 5 * nnr * math.log2(nnr) + 16 * ngw * 4 * nat)
    return dict(bytes=data, flops=applications * flops)


def work(case):
    kind = case["kind"]
    if kind == "hpsi":
        return _hpsi_work(case, case["nb"])
    if kind == "filter":
        return _hpsi_work(case, case["nb"], case["degree"])
    if kind == "batch":
        parts = [_hpsi_work(sub, sub["nb"]) for sub in _batch_cases(case)]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    if kind == "eig":
        n = case["n"]
        return dict(bytes=2 * 16 * n * n + 8 * n, flops=4 * (4 / 3 + 2) * n ** 3)
    ngw, nnr, nat = _estimate(case)
    if kind == "rho":
        return dict(bytes=case["nb"] * ngw * 16 + nnr * 8,
                    flops=case["nb"] * (5 * nnr * math.log2(nnr) + 4 * nnr))
    if kind == "ortho":
        return dict(bytes=2 * case["nb"] * ngw * 16, flops=8 * case["nb"] ** 2 * ngw)
    # per SCF iteration: filter, orthonormalisation, Rayleigh-Ritz, density, projections
    nb = 2 * nat + case["nempty"] + 2
    one = nb * (11 * (2 * 5 * nnr * math.log2(nnr) + 16 * ngw * 4 * nat)
                + 5 * nnr * math.log2(nnr) + 8 * ngw * 4 * nat) + 8 * nb * nb * ngw * 4
    return dict(bytes=ngw * (nat * 16 + 40) + 8 * nnr, flops=case["iters"] * one)


# ---------------------------------------------------------------- 64-bit values
def _exact_hpsi(b, veff):
    """H as a function on blocks (bands in rows), with dense projectors."""
    ngw, (n1, n2, n3) = b["ngw"], b["nr"]
    idx = torch.tensor(np.asarray(b["n123"][:ngw], dtype=np.int64) - 1, device=DEV)
    kin = torch.tensor(0.5 * np.asarray(b["xkg"][:ngw]) * b["tpiba2"], device=DEV)
    eigr = torch.tensor(np.ascontiguousarray(b["eigr"][:ngw, :, 0]), device=DEV)
    pkg = torch.tensor(np.ascontiguousarray(b["pkg_a"][:, :ngw, 0]), device=DEV)
    beta = (eigr[:, :, None] * pkg.T[:, None, :]).reshape(ngw, -1)
    w = torch.tensor(np.asarray(b["wnl"])[0], device=DEV).repeat(eigr.shape[1])
    v = veff.reshape(n3, n2, n1)

    def apply(x):
        out = kin[None] * x + ((x @ beta.conj()) * w[None]) @ beta.T
        step = max(1, (1 << 25) // veff.numel())
        for i in range(0, len(x), step):
            part = x[i:i + step]
            box = torch.zeros(len(part), veff.numel(), device=DEV, dtype=torch.complex128)
            box[:, idx] = part
            box = torch.fft.ifftn(box.reshape(-1, n3, n2, n1), dim=(1, 2, 3)) * v
            out[i:i + step] += torch.fft.fftn(box, dim=(1, 2, 3)).reshape(len(part), -1)[:, idx]
        return out

    return apply


def _exact_filter(apply, x, degree, lb, ub):
    """The scaled three-term Chebyshev recurrence of chebyfilt.cpp:8-67."""
    e, c = (ub - lb) / 2.0, (ub + lb) / 2.0
    sigma = e / (lb - ub)
    sigma1 = sigma
    prev, cur = x, (apply(x) - c * x) * (sigma1 / e)
    for _ in range(2, degree + 1):
        s2 = 1.0 / (2.0 / sigma1 - sigma)
        prev, cur = cur, (apply(cur) - c * cur) * (2.0 * s2 / e) - prev * (sigma * s2)
        sigma = s2
    return cur


def exact(case, seed):
    kind = case["kind"]
    if kind == "scf":
        return None
    if kind == "eig":
        return dict(vectors=None, values=torch.linalg.eigvalsh(_dense_hermitian(case["n"], seed)))
    if kind == "batch":
        outs = []
        for i, sub in enumerate(_batch_cases(case)):
            b, veff, x, _ = _cell_inputs(sub, seed + 1000 * i)
            outs.append(_exact_hpsi(b, veff)(x.to(torch.complex128)))
        return outs
    b, veff, x, g = _cell_inputs(case, seed)
    if kind == "ortho":
        m = torch.randn(len(x), len(x), 2, generator=g, device=DEV, dtype=torch.float64)
        q, r = torch.linalg.qr((torch.view_as_complex(m) @ x).T)
        d = torch.diagonal(r)
        return (q * (d / d.abs())[None]).T.contiguous()
    if kind == "rho":
        nb, ngw = x.shape
        n1, n2, n3 = b["nr"]
        f = torch.tensor(np.where(np.arange(nb) < max(1, (9 * nb) // 10), 2.0, 0.0), device=DEV)
        x = x[:, :ngw - 1]  # the reference leaves out the last plane wave
        idx = torch.tensor(np.asarray(b["n123"][:ngw - 1], dtype=np.int64) - 1, device=DEV)
        xkg = torch.tensor(np.asarray(b["xkg"][:ngw - 1]), device=DEV)
        rho = torch.zeros(veff.numel(), device=DEV, dtype=torch.float64)
        for i in range(nb):
            box = torch.zeros(veff.numel(), device=DEV, dtype=torch.complex128)
            box[idx] = x[i]
            psi = torch.fft.ifftn(box.reshape(n3, n2, n1), norm="forward").reshape(-1)
            rho += f[i] / b["omega"] * (psi.real ** 2 + psi.imag ** 2)
        ekin = 0.5 * (f[:, None] * xkg[None] * (x.real ** 2 + x.imag ** 2)).sum() * b["tpiba2"]
        return dict(rho=rho, ekin=float(ekin))
    apply = _exact_hpsi(b, veff)
    x = x.to(torch.complex128)
    return apply(x) if kind == "hpsi" else _exact_filter(apply, x, case["degree"], LB, UB)
