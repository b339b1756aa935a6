"""Plaintext-matrix times ciphertext with the diagonals resident in HBM (no counterpart in the reference).

The reference's bsgs_matmul_preencoded (src/bsgs.cu:194-367, mirrored by pyPhantom.bsgs_matmul_preencoded) keeps
every diagonal as one int64 tower on the host and, for every giant step of every product, copies M of them to the
device and expands and transforms them again; its babies are a chain of dependent rotations and its giants a Horner
chain of dependent rotations. On a GPU with 180 GB of HBM the expanded diagonals of a 4096 x 4096 matrix at 16 limbs
(32 GB) simply stay resident, and the product becomes:

  babies   rot(x, b), b = 1 .. M-1     one hoisted call, one ModUp
  partials sum_b pt[g][b] * baby_b      four giants per launch, every baby read once per launch
  giants   sum_g rot(partial_g, g*M)    decomposed together, inner products summed in one launch, one ModDown
  one rescale, scale reset to the input's

It needs a Galois key for every baby step 1..M-1 and every giant step M, 2M, .. (G-1)M (the "64 + 64 keys" form);
the result decrypts to the same product as the reference's driver but is not limb-identical to it (hoisted babies).
Babies and partial sums live in buffers of the plan: two products of one plan belong on one stream, or the second waits for the
first; concurrent ones take a plan each.
"""
import numpy as np
import torch

from . import _native, get_elt_from_step, rescale_to_next
from ._native import LIB, check, current_stream as _stream


class resident_bsgs:
    def __init__(self, context, galois_key_, diags, chain_index):
        ctx = self.ctx = context
        self.M, self.G, self.d_pad = diags.baby_steps, diags.giant_steps, diags.d_pad
        if self.M * self.G != self.d_pad or len(diags.diagonals) != self.d_pad:
            raise ValueError("resident_bsgs: M*G must equal d_pad and every diagonal must be present")
        self.chain_index, self.l = chain_index, ctx.limbs_at(chain_index)
        self.pt_scale = diags.diagonals[0].scale
        l, N, M, G = self.l, ctx.N, self.M, self.G
        # expand every diagonal once: [d_pad][l][N], NTT form
        self.pts = ctx.empty(self.d_pad, l)
        for d, scp in enumerate(diags.diagonals):
            if scp.coeffs.numel() != N:
                raise ValueError("resident_bsgs: scp coeff length != N")
            stage = scp.coeffs.to(ctx.device, non_blocking=True)
            check(LIB.b2_expand_single_chain(ctx._h, l, stage.data_ptr(), self.pts[d].data_ptr(), _stream()))
        # keys by step
        self.keys = {}
        for s in list(range(1, M)) + [g * M for g in range(1, G)]:
            e = get_elt_from_step(s, N)
            if e not in ctx.galois_elts:
                raise ValueError(f"resident_bsgs: no Galois element for step {s} in the context")
            k = galois_key_.resolve(ctx.galois_elts.index(e))
            if k is None:
                raise ValueError(f"resident_bsgs: no Galois key for step {s}")
            self.keys[s] = (e, k)
        self.baby_buf = ctx.empty(M, 2, l)
        self.part_buf = ctx.empty(G, 2, l)
        self.baby_tab = torch.tensor([self.baby_buf[b].data_ptr() for b in range(M)], dtype=torch.int64, device=ctx.device)
        # giants four to a launch; giant 0 (no rotation) is the sum the others are added to
        self.groups = []
        for g0 in range(0, G, 4):
            chunk = range(g0, min(G, g0 + 4))
            tab = np.array([[self.pts[g * M + b].data_ptr() for b in range(M)] for g in chunk], dtype=np.int64)
            self.groups.append((len(chunk), torch.from_numpy(tab.ravel().copy()).to(ctx.device),
                                torch.tensor([self.part_buf[g].data_ptr() for g in chunk], dtype=torch.int64, device=ctx.device)))
        self.baby_steps, self.giant_steps = range(1, M), range(M, M * G, M)
        self.baby_elts, self.giant_elts = (np.array([self.keys[s][0] for s in steps], dtype=np.uint32) for steps in (self.baby_steps, self.giant_steps))
        self.baby_outs = np.array([self.baby_buf[b].data_ptr() for b in range(1, M)], dtype=np.uint64)
        torch.cuda.synchronize()

    def _digits(self, steps, n_evk):
        """the addresses of the first n_evk digits of every step's key, as they are at this call (a key may be loaded anew)"""
        if any(self.keys[s][1].dnum() < n_evk for s in steps):
            raise ValueError("key has fewer digits than this level needs")
        return np.concatenate([self.keys[s][1].pointer_table()[:n_evk] for s in steps]).astype(np.uint64)

    def apply(self, x):
        ctx, l, N, M = self.ctx, self.l, self.ctx.N, self.M
        if x._chain_index != self.chain_index or x._size != 2:
            raise ValueError("resident_bsgs: the ciphertext is not at the level the diagonals were expanded for")
        n_evk, st = ctx.beta(l), _stream()
        self.baby_buf[0].copy_(x.data)
        if M > 1:
            ws, nbytes = ctx.workspace(_native.OP_HOIST, l)
            ksk = self._digits(self.baby_steps, n_evk)
            check(LIB.b2_hoist_rotations(ctx._h, l, x.data.data_ptr(), self.baby_elts.ctypes.data, M - 1, ksk.ctypes.data, n_evk,
                                         self.baby_outs.ctypes.data, ws.data_ptr(), nbytes, st))
        for n, ptab, otab in self.groups:
            check(LIB.b2_bsgs_mac_multi(ctx._h, l, M, n, ptab.data_ptr(), self.baby_tab.data_ptr(), otab.data_ptr(), st))
        total = self.part_buf[0]
        if self.G > 1:
            n = self.G - 1
            nbytes = int(LIB.b2_rotate_sum_workspace_bytes(ctx._h, l, n))
            ws = torch.empty(nbytes // 8, dtype=torch.int64, device=ctx.device)
            ksk = self._digits(self.giant_steps, n_evk)
            check(LIB.b2_rotate_sum(ctx._h, l, n, self.giant_elts.ctypes.data, self.part_buf[1].data_ptr(), 2 * l, ksk.ctypes.data, n_evk,
                                    total.data_ptr(), 0, ws.data_ptr(), nbytes, st))
        out = rescale_to_next(ctx, x._like(total, scale=x._scale * self.pt_scale))
        out.set_scale(x._scale)
        return out
