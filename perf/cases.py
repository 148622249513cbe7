"""Performance cases: the calls a quantum-chemistry program makes on a built
representation of the electron-repulsion integrals (ERI).

A self-consistent-field program builds the representation once per geometry
and then asks for Coulomb (J) and exchange (K) matrices of one density after
another. So the representation is what such a program keeps (one per geometry,
tolerance and precision, shared by every density of this process), and a
case's inputs are its densities or vectors.

Fields of a case:
  call   what is called: "coulomb", "exchange", "matvec", "batch"
  mol    geometry: "alkane:N" (all-trans C_N H_2N+2) or "methane:AxBxC" (CH4 on
         a jittered lattice, a 3-D system); "alkane:8,13,..." for a batch
  tol    QR tolerance of the representation
  mode   "fp64" (the default precision) or "mixed" (FP32 blocks, J to 1e-8)
  n      densities (or vectors) per call
  where  "host": numpy arrays in and out, as a reference caller has them;
         "device": CUDA arrays, enqueued on the caller's stream
"""
import atexit
import ctypes
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "h2p-eri_gb300"))

import h2eri_gb300 as hg  # noqa: E402
from h2eri_gb300 import molecules  # noqa: E402


def listed():
    return [
        # smallest call: J of ethane through the reference's calling sequence,
        # numpy in and out; launches and host latency decide
        dict(name="coulomb_host_c2_fp64", call="coulomb", mol="alkane:2", tol=1e-6, mode="fp64", n=1, where="host"),
        # an ordinary molecule in the default precision, host arrays: the
        # benchmark's CPU-runnable configuration (C10H22, 1e-6)
        dict(name="coulomb_host_c10_fp64", call="coulomb", mol="alkane:10", tol=1e-6, mode="fp64", n=1, where="host"),
        # the benchmark molecule in the default precision
        dict(name="coulomb_c30_fp64", call="coulomb", mol="alkane:30", tol=1e-8, mode="fp64", n=1, where="device"),
        # the benchmark's headline: one density per call, mixed precision
        dict(name="coulomb_c30_mixed", call="coulomb", mol="alkane:30", tol=1e-8, mode="mixed", n=1, where="device"),
        # stacked trial densities in one call
        dict(name="coulomb_c30_mixed_n16", call="coulomb", mol="alkane:30", tol=1e-8, mode="mixed", n=16, where="device"),
        # the largest molecule of the benchmark
        dict(name="coulomb_c100_mixed", call="coulomb", mol="alkane:100", tol=1e-8, mode="mixed", n=1, where="device"),
        # the bare operator on a few vectors at once (alpha and beta densities
        # and response vectors), default precision, odd molecule size
        dict(name="matvec_c13_fp64_n5", call="matvec", mol="alkane:13", tol=1e-7, mode="fp64", n=5, where="device"),
        # many molecules of uneven size in one call, alpha and beta densities
        dict(name="batch_mixed_n2", call="batch", mol="alkane:8,13,21,30,11", tol=1e-8, mode="mixed", n=2,
             where="device"),
        # K of a small molecule, default precision, host arrays
        dict(name="exchange_host_c5_fp64", call="exchange", mol="alkane:5", tol=1e-6, mode="fp64", n=1, where="host"),
        # K of an ordinary molecule, default precision
        dict(name="exchange_c10_fp64", call="exchange", mol="alkane:10", tol=1e-6, mode="fp64", n=1, where="device"),
        # K of the benchmark molecule, mixed precision
        dict(name="exchange_c30_mixed", call="exchange", mol="alkane:30", tol=1e-8, mode="mixed", n=1, where="device"),
        # K of a 3-D cluster, mixed precision
        dict(name="exchange_ch4x8_mixed", call="exchange", mol="methane:2x2x2", tol=1e-7, mode="mixed", n=1,
             where="device"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: chains of 1 to 60 carbons for J and the bare
    operator, 1 to 24 (mixed) or 12 (FP64) for K, clusters of up to 12 CH4,
    1 to 16 densities per call, the three tolerances in use."""
    call = rng.choice(["coulomb", "coulomb", "coulomb", "exchange", "exchange", "matvec", "batch"])
    mode = rng.choice(["fp64", "mixed"])
    tol = rng.choice([1e-6, 1e-7, 1e-8])
    where = rng.choice(["host", "device", "device"])
    n = rng.choice([1, 1, _log_int(rng, 1, 16)])
    mol = "alkane:%d" % _log_int(rng, 1, 60)
    if call == "exchange":
        mol = "alkane:%d" % _log_int(rng, 1, 24 if mode == "mixed" else 12)
        if rng.random() < 0.3:
            mol = "methane:%dx%dx%d" % (rng.randint(1, 2), rng.randint(1, 2), rng.randint(2, 3))
        n, where = 1, rng.choice(["host", "device"])
    elif call == "batch":
        mode, n, where = "mixed", rng.choice([1, 2, 2, 3]), "device"
        mol = "alkane:" + ",".join(str(k) for k in rng.sample(range(2, 31), rng.randint(2, 4)))
    elif mode == "fp64" and n > 4:
        mol = "alkane:%d" % _log_int(rng, 1, 30)
    return dict(call=call, mol=mol, tol=tol, mode=mode, n=n, where=where)


# --------------------------------------------------------------------------
# representations: one per geometry, tolerance and precision
# --------------------------------------------------------------------------

_handles = {}


@atexit.register
def _release():
    for h in _handles.values():
        h.destroy()
    _handles.clear()


def _members(case):
    kind, _, size = case["mol"].partition(":")
    return ["%s:%s" % (kind, s) for s in size.split(",")]


def _handle(mol, tol, mode, upload=True):
    key = (mol, tol, mode)
    if key not in _handles:
        kind, _, size = mol.partition(":")
        with tempfile.TemporaryDirectory() as d:
            path = os.path.join(d, "m.mol")
            if kind == "alkane":
                molecules.write_alkane(path, int(size))
            else:
                molecules.write_methane_cluster(path, shape=tuple(int(s) for s in size.split("x")))
            _handles[key] = hg.H2ERI.from_mol(path, qr_tol=tol)
    h = _handles[key]
    if upload:
        h.upload()
        h.set_precision(hg.MIXED if mode == "mixed" else hg.FP64)
    return h


def _n_occ(mol):
    kind, _, size = mol.partition(":")
    if kind == "alkane":
        return 4 * int(size) + 1
    return 5 * math.prod(int(s) for s in size.split("x"))


def _densities(case, seed, mol, nbf):
    """[n][nbf][nbf]: projectors on random orthonormal orbitals."""
    k = _members(case).index(mol)
    return np.stack([molecules.seeded_density(nbf, min(_n_occ(mol), nbf), [seed, k, i]) for i in range(case["n"])])


def _vectors(case, seed, size):
    return np.random.default_rng(seed).standard_normal((case["n"], size))


# --------------------------------------------------------------------------
# the calls
# --------------------------------------------------------------------------

_streams = []


def _stream():
    """The program's own stream (the library's streams are non-blocking)."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return ctypes.c_void_p(_streams[0].cuda_stream)


def _ok(rc):
    if rc != 0:
        raise hg.H2ERIError(hg.lib().H2ERI_gpu_last_error().decode())


def prepare(case, seed):
    st = dict(case=case, h=[_handle(m, case["tol"], case["mode"]) for m in _members(case)])
    if case["call"] == "matvec":
        ins = [_vectors(case, seed, st["h"][0].krnl_mat_size)]
    else:
        ins = [_densities(case, seed, m, h.num_bf) for m, h in zip(_members(case), st["h"])]
    if case["where"] == "host":
        st["in"] = [x[0] if case["n"] == 1 else x for x in ins]
    else:
        st["in"] = [torch.from_numpy(x).cuda() for x in ins]
        st["out"] = [torch.empty_like(x) for x in st["in"]]
        if case["call"] == "batch":
            m = len(ins)
            st["args"] = (m, (ctypes.c_void_p * m)(*[h.handle.value for h in st["h"]]), (ctypes.c_int * m)(*[case["n"]] * m),
                          (ctypes.c_void_p * m)(*[x.data_ptr() for x in st["in"]]),
                          (ctypes.c_void_p * m)(*[x.data_ptr() for x in st["out"]]))
    return st


def run(st):
    case, h, L = st["case"], st["h"][0], hg.lib()
    if case["where"] == "host":
        call = {"coulomb": h.build_coulomb, "exchange": h.build_exchange, "matvec": h.matvec}[case["call"]]
        return call(st["in"][0])
    if case["call"] == "batch":
        _ok(L.H2ERI_build_Coulomb_batch(*st["args"], _stream()))
        return st["out"]
    x, y = st["in"][0].data_ptr(), st["out"][0].data_ptr()
    if case["call"] == "coulomb":
        _ok(L.H2ERI_build_Coulomb_device(h.handle, case["n"], x, y, _stream()))
    elif case["call"] == "matvec":
        _ok(L.H2ERI_matvec_device(h.handle, case["n"], x, y, _stream()))
    else:
        _ok(L.H2ERI_build_exchange_device(h.handle, x, y, _stream()))
    return st["out"][0]


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def _work(case, mol):
    h = _handle(mol, case["tol"], case["mode"], upload=False)
    s = h.s
    nbf, n, leaf = h.num_bf, case["n"], s.n_leaf_node
    size = {}
    for kind, cnt, ptr in (("U", s.n_UJ, s.U), ("B", s.n_B, s.c_B_blks), ("D", s.n_D, s.c_D_blks)):
        arr = ctypes.cast(ptr, ctypes.POINTER(ctypes.POINTER(hg.DenseMat)))
        size[kind] = [(m.nrow + m.ncol) * -m.ld if m.ld < 0 else m.nrow * m.ncol
                      for m in (arr[i].contents for i in range(cnt))]
    u, b, diag, d = sum(size["U"]), sum(size["B"]), sum(size["D"][:leaf]), sum(size["D"][leaf:])
    width = (8, 8, 4, 4) if case["mode"] == "mixed" else (8, 8, 8, 8)   # U, leaf D, B, other D
    stored = u * width[0] + diag * width[1] + b * width[2] + d * width[3]
    if case["call"] == "exchange":
        out = np.zeros(8)
        _ok(hg.lib().H2ERI_exchange_plan_check(h.handle, 80e9, out.ctypes.data, 8))
        return stored + n * 16 * nbf * nbf, n * float(out[0])
    io = 16 * (h.krnl_mat_size if case["call"] == "matvec" else nbf * nbf)
    return stored + n * io, n * (4.0 * u + 4.0 * b + 2.0 * diag + 4.0 * d)


def work(case):
    """Every stored block read once, every density or vector read and every
    result written once; the products of one application of the blocks (for K
    those of its transforms, couplings and near field)."""
    w = [_work(case, m) for m in _members(case)]
    return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}


# --------------------------------------------------------------------------
# the same results from the stored blocks in 64 bits, in plain torch
# --------------------------------------------------------------------------

class _Plain:
    """The stored representation (its U, B and D blocks and its tree) as
    float64 tensors, applied block by block."""

    def __init__(self, h):
        s = h.s
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        ints = h.int_array
        self.dev, self.n, self.nbf, self.n_node = dev, h.krnl_mat_size, h.num_bf, s.n_node
        self.first = ints("mat_cluster", 2 * s.n_node)[0::2]
        self.size = ints("mat_cluster", 2 * s.n_node)[1::2] - self.first + 1
        self.n_child = ints("n_child", s.n_node)
        self.child = ints("children", s.n_node * s.max_child).reshape(s.n_node, s.max_child)
        self.level = ints("node_level", s.n_node)
        self.max_level, self.min_adm = s.max_level, s.min_adm_level
        self.leaves = ints("height_nodes", s.n_leaf_node)
        self.adm = ints("r_adm_pairs", 2 * s.n_r_adm_pair).reshape(-1, 2)
        self.inadm = ints("r_inadm_pairs", 2 * s.n_r_inadm_pair).reshape(-1, 2)
        self.U = [(r, c, torch.from_numpy(d.reshape(r, c)).to(dev)) for r, c, _, d in h.blocks("U")]
        self.B = [self._block(*b) for b in h.blocks("B")]
        self.D = [self._block(*b) for b in h.blocks("D")]
        # function pair of every vector entry
        sp = ints("sp_shell_idx", 2 * s.num_sp).reshape(2, s.num_sp)
        bf, start = ints("shell_bf_sidx", s.nshell + 1), ints("sp_bfp_sidx", s.num_sp + 1)
        self.row = np.zeros(self.n, np.int64)     # function of the second shell
        self.col = np.zeros(self.n, np.int64)     # function of the first shell
        self.same = np.zeros(self.n, bool)
        for i in range(s.num_sp):
            m, k = sp[0, i], sp[1, i]
            nm, nk = bf[m + 1] - bf[m], bf[k + 1] - bf[k]
            e = slice(start[i], start[i] + nm * nk)
            self.row[e] = np.repeat(np.arange(bf[k], bf[k + 1]), nm)
            self.col[e] = np.tile(np.arange(bf[m], bf[m + 1]), nk)
            self.same[e] = m == k
        self.row, self.col, self.same = (torch.from_numpy(a).to(dev) for a in (self.row, self.col, self.same))

    def _block(self, nrow, ncol, ld, data):
        t = torch.from_numpy(data).to(self.dev)
        if ld < 0:
            return t[:nrow * -ld].reshape(nrow, -ld), t[nrow * -ld:].reshape(ncol, -ld)
        return t.reshape(nrow, ncol), None

    @staticmethod
    def _mul(b, x):
        return b[0] @ x if b[1] is None else b[0] @ (b[1].T @ x)

    @staticmethod
    def _mul_t(b, x):
        return b[0].T @ x if b[1] is None else b[1] @ (b[0].T @ x)

    def apply(self, x):
        """A x for the columns of x."""
        y = torch.zeros_like(x)

        def span(i):
            return slice(self.first[i], self.first[i] + self.size[i])

        y0, y1 = [None] * self.n_node, [0.0] * self.n_node
        for lv in range(self.max_level, self.min_adm - 1, -1):
            for i in np.flatnonzero(self.level == lv):
                r, c, u = self.U[i]
                if c == 0:
                    y0[i] = x[:0]
                elif self.n_child[i] == 0:
                    y0[i] = u.T @ x[span(i)]
                else:
                    y0[i] = u.T @ torch.cat([y0[k] for k in self.child[i, :self.n_child[i]]])
        for (i, j), b in zip(self.adm, self.B):
            if b[0].numel() == 0:
                continue
            up_i, up_j = self.level[i] >= self.level[j], self.level[j] >= self.level[i]
            to_i = self._mul(b, y0[j] if up_j else x[span(j)])
            to_j = self._mul_t(b, y0[i] if up_i else x[span(i)])
            for k, up, v in ((i, up_i, to_i), (j, up_j, to_j)):
                if up:
                    y1[k] = y1[k] + v
                else:
                    y[span(k)] += v
        for lv in range(self.min_adm, self.max_level + 1):
            for i in np.flatnonzero(self.level == lv):
                if isinstance(y1[i], float) or self.U[i][1] == 0:
                    continue
                t = self.U[i][2] @ y1[i]
                if self.n_child[i] == 0:
                    y[span(i)] += t
                    continue
                at = 0
                for k in self.child[i, :self.n_child[i]]:
                    y1[k] = y1[k] + t[at:at + self.U[k][1]]
                    at += self.U[k][1]
        for i, b in zip(self.leaves, self.D):
            y[span(i)] += self._mul(b, x[span(i)])
        for (i, j), b in zip(self.inadm, self.D[len(self.leaves):]):
            if b[0].numel():
                y[span(i)] += self._mul(b, x[span(j)])
                y[span(j)] += self._mul_t(b, x[span(i)])
        return y

    def coulomb(self, den):
        den = torch.from_numpy(den).to(self.dev)
        x = den[:, self.row, self.col] * torch.where(self.same, 1.0, 2.0)
        y = self.apply(x.T.contiguous()).T * torch.where(self.same, 0.5, 1.0)
        J = torch.zeros_like(den)
        J[:, self.row, self.col] = y
        return J + J.transpose(1, 2)

    def exchange(self, den):
        """K[m][q] = sum_np A[(m n), (p q)] D[n][p] with the operator formed in full."""
        n, nbf, dev = self.n, self.nbf, self.dev
        A = torch.empty(n, n, dtype=torch.float64, device=dev)
        for c in range(0, n, 2048):
            w = min(2048, n - c)
            e = torch.zeros(n, w, dtype=torch.float64, device=dev)
            e[torch.arange(c, c + w, device=dev), torch.arange(w, device=dev)] = 1.0
            A[:, c:c + w] = self.apply(e)
        at = torch.full((nbf, nbf), -1, dtype=torch.int64, device=dev)
        at[self.row, self.col] = torch.arange(n, device=dev)
        at = torch.where(at < 0, at.T, at)
        at[self.row[self.same], self.col[self.same]] = torch.arange(n, device=dev)[self.same]
        D = torch.from_numpy(den[0]).to(dev)
        K = torch.zeros_like(D)
        # every (p, q) that holds a pair, sorted by q for the segmented sums
        q, p = torch.nonzero(at.T >= 0, as_tuple=True)
        c = at[p, q]
        for m in range(nbf):
            nn = torch.nonzero(at[m] >= 0)[:, 0]
            W = D[nn].T @ A[at[m, nn]]               # [p][pair]
            K[m] = torch.zeros(nbf, dtype=torch.float64, device=dev).index_add_(0, q, W[p, c])
        return K


def exact(case, seed):
    hs = [_handle(m, case["tol"], case["mode"], upload=False) for m in _members(case)]
    if case["call"] == "exchange" and hs[0].krnl_mat_size > 50000:
        return None      # the operator in full takes too long
    plain = [_Plain(h) for h in hs]
    if case["call"] == "matvec":
        x = torch.from_numpy(_vectors(case, seed, plain[0].n)).to(plain[0].dev)
        y = plain[0].apply(x.T.contiguous()).T.contiguous()
        return y if case["n"] > 1 or case["where"] == "device" else y[0]
    dens = [_densities(case, seed, m, h.num_bf) for m, h in zip(_members(case), hs)]
    if case["call"] == "exchange":
        K = plain[0].exchange(dens[0])
        return K if case["where"] == "host" else K[None]
    J = [p.coulomb(d) for p, d in zip(plain, dens)]
    if case["call"] == "batch":
        return J
    return J[0] if case["where"] == "device" or case["n"] > 1 else J[0][0]
