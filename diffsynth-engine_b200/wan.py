"""One Wan2.1-architecture DiT denoising step on the library's kernels (the job of ``WanDiT.forward``,
models/wan/wan_dit.py:319-351 of DiffSynth-Engine, text-to-video, batch 1), optionally sequence-parallel over
the ranks of a ``torch.distributed`` group (Ulysses):

  * every rank owns a contiguous slice of S/P tokens in (f, h, w) raster order and runs all token-wise work on
    it: AdaLN, every Linear, the full-width QK-RMSNorm, RoPE with the slice's own positions, cross-attention
    (queries of the slice against the replicated 512-token context), FFN;
  * self-attention needs one exchange on each side: q, k, v go from ``[S/P, H, 128]`` to ``[S, H/P, 128]`` (all
    tokens, this rank's heads) and the attention output goes back.  The RMSNorm/RoPE kernel writes q and k straight
    into the per-peer-contiguous send layout ``[P][S/P][H/P*128]``, and the quantiser that feeds the output
    projection reads the returned ``[P][S/P][H/P*128]`` directly, so neither direction needs a pack kernel;
  * the exchanges run on a second stream, each as soon as its send layout is written; weights (14 GB in FP8) are
    replicated;
  * with ``exchange="peer"`` (the default when the ranks can map each other's memory) only k and v travel that way:
    the attention kernel itself reads the queries of each token range from the rank that owns it and writes each
    output row into the memory of the rank that owns the token (``dsb_flash_attn_parts`` over peer pointers), with
    one ``dsb_rank_barrier`` before and after it - the exchanges of q and of the attention output cost no launch
    and no exposed time.

Per block, in launch order:
  P = 1: ln_modulate+quantise -> ONE q|k|v GEMM (N = 3d) -> rmsnorm_full+rope of q, of k -> flash attention
  P > 1: ln_modulate+quantise -> k GEMM -> rmsnorm_full+rope of k -> [a2a k] | v GEMM -> v re-layout -> [a2a v]
         | q GEMM -> rmsnorm_full+rope of q -> (peer: rank barrier | nccl: [a2a q]) -> flash attention (H/P heads,
         all tokens; peer: queries read from, output rows written to, the owning ranks) -> (peer: rank barrier |
         nccl: [a2a o])
  then: quantise -> o GEMM with x += gate*(.) -> affine LN3+quantise -> q GEMM -> rmsnorm_full
  -> flash attention (Sk = context; keys and values of the context are cached per prompt) -> quantise
  -> o GEMM with x += (.) -> ln_modulate+quantise -> FFN GEMM (+GELU) -> quantise -> FFN GEMM with x += gate*(.)
"""
from typing import Dict, Optional

import torch

from . import ops
from .packed import PackedLinear, act_format, pack_linear


def wan_rope_table(f: int, h: int, w: int, head_dim: int = 128, theta: float = 10000.0, device="cpu") -> torch.Tensor:
    """(cos, sin) per rotated pair for the (f, h, w) grid in raster order, fp32 [f*h*w, 64, 2]; angles in fp64 and the
    44/42/42 split of the 128 head dims as models/wan/wan_dit.py:38-51,335-346 build them."""
    def freqs(dim, end):
        fr = 1.0 / (theta ** (torch.arange(0, dim, 2, device=device)[: dim // 2].double() / dim))
        return torch.outer(torch.arange(end, dtype=torch.float64, device=device), fr)

    d_h = head_dim // 3
    d_f = head_dim - 2 * d_h
    ang = torch.cat([
        freqs(d_f, f).view(f, 1, 1, -1).expand(f, h, w, -1),
        freqs(d_h, h).view(1, h, 1, -1).expand(f, h, w, -1),
        freqs(d_h, w).view(1, 1, w, -1).expand(f, h, w, -1),
    ], dim=-1).reshape(f * h * w, -1)
    return torch.stack([torch.cos(ang), torch.sin(ang)], dim=-1).float().contiguous()


IMG_TOKENS = 257   # CLIP tokens at the head of an image-to-video context (wan_dit.py:138-139)


def _stack_linears(parts):
    """Row-stack Linears that read the same activation (self-attention q, k, v; wan_dit.py:85-87) into one
    ``[sum N, K]`` weight with a per-row scale, so one GEMM launch serves them all."""
    fmt = parts[0].fmt
    w = torch.cat([p.w for p in parts], dim=0).contiguous()
    scale = None
    if fmt != "bf16":
        scale = torch.cat([p.scale if p.scale.numel() > 1 else p.scale.expand(p.w.shape[0]) for p in parts]).contiguous()
    bias = torch.cat([p.bias for p in parts]).contiguous()
    return PackedLinear(w, scale, bias, fmt)


class HeadExchange:
    """The Ulysses all-to-all.  ``send`` is ``[P, rows, C]``: chunk p goes to rank p; the result's chunk r came from
    rank r.  Forward (tokens -> heads): rows = S/P own tokens, chunk p = head group p; result = all S tokens of the
    own head group.  Backward (heads -> tokens) is the same call on the attention output viewed ``[P, S/P, C]``."""

    def __init__(self, group=None):
        import torch.distributed as dist
        self.dist = dist
        self.group = group
        self.world = dist.get_world_size(group) if dist.is_initialized() else 1
        self.rank = dist.get_rank(group) if dist.is_initialized() else 0

    def __call__(self, send: torch.Tensor, recv: Optional[torch.Tensor] = None) -> torch.Tensor:
        if self.world == 1:
            return send
        if recv is None:
            recv = torch.empty_like(send)
        self.dist.all_to_all_single(recv, send, group=self.group)
        return recv


class PeerMemory:
    """One device buffer per rank, mapped into the address space of every rank of the group (torch symmetric memory:
    CUDA virtual-memory handles exchanged through the group's store).  ``ptrs[r]`` is rank r's buffer as this
    process addresses it; ``local`` is this rank's own buffer as a uint8 tensor.  Binding the buffers to an NVLink
    multicast object is switched off: only plain peer loads and stores are used here, and a rank that dies while
    bound takes the other ranks' GPUs with it."""

    def __init__(self, nbytes: int, device, group):
        import os
        os.environ.setdefault("TORCH_SYMM_MEM_DISABLE_MULTICAST", "1")
        import torch.distributed._symmetric_memory as symm
        self.local = symm.empty(nbytes, dtype=torch.uint8, device=device)
        self.local.zero_()
        self.handle = symm.rendezvous(self.local, group)
        self.ptrs = [int(p) for p in self.handle.buffer_ptrs]
        if len(self.ptrs) != self.handle.world_size or self.ptrs[self.handle.rank] != self.local.data_ptr():
            raise RuntimeError("symmetric memory handle does not describe this group")


class WanDiTEngine:
    def __init__(self, state_dict: Dict[str, torch.Tensor], fmt: str = "fp8_channel", device="cuda:0",
                 num_layers: int = 40, num_heads: int = 40, eps: float = 1e-6, freq_dim: int = 256, group=None,
                 release_source: bool = False, overlap: bool = True, exchange: str = "auto", tail_split: bool = True):
        self.dev = torch.device(device)
        self.fmt, self.afmt = fmt, act_format(fmt)
        self.L, self.H, self.eps, self.freq_dim = num_layers, num_heads, eps, freq_dim
        self.xchg = HeadExchange(group)
        # without a group the engine is a one-GPU replica even inside an initialised process group
        self.P, self.rank = (self.xchg.world, self.xchg.rank) if group is not None else (1, 0)
        if group is None:
            self.xchg.world, self.xchg.rank = 1, 0
        if num_heads % self.P:
            raise ValueError(f"{num_heads} heads do not split over {self.P} ranks")
        sd = state_dict
        self.d = sd["time_embedding.0.weight"].shape[0]
        if self.d // num_heads != 128:
            raise ValueError("head_dim must be 128")
        self.overlap = overlap and self.P > 1
        # how q and the attention output cross ranks: "nccl" = all-to-all like k and v; "peer" = inside the attention
        # kernel over mapped peer memory; "auto" = peer when the mapping can be set up (decided in prepare)
        if exchange not in ("auto", "peer", "nccl"):
            raise ValueError("exchange must be 'auto', 'peer' or 'nccl'")
        self.exchange = "nccl" if self.P == 1 else exchange
        self._group = group
        self._epoch = 0
        # peer mode: let the attention kernel cut the items of a partly filled last wave along the keys (the cut rows
        # then differ from an uncut evaluation in fp32 summation order)
        self.tail_split = tail_split

        def P_(name):
            p = pack_linear(sd[name + ".weight"], sd.get(name + ".bias"), fmt, self.dev)
            if release_source:
                sd.pop(name + ".weight", None), sd.pop(name + ".bias", None)
            return p

        def V(name):
            v = sd[name].to(device=self.dev, dtype=torch.float32).contiguous()
            if release_source:
                sd.pop(name, None)
            return v

        self.patch = P_("patch_embedding")
        self.text0, self.text2 = P_("text_embedding.0"), P_("text_embedding.2")
        self.time0, self.time2, self.tproj = P_("time_embedding.0"), P_("time_embedding.2"), P_("time_projection.1")
        self.blocks = []
        mods = []
        for i in range(num_layers):
            pre = f"blocks.{i}."
            mods.append(V(pre + "modulation").reshape(6, self.d))
            self.blocks.append(dict(
                sq=P_(pre + "self_attn.q"), sk=P_(pre + "self_attn.k"), sv=P_(pre + "self_attn.v"),
                so=P_(pre + "self_attn.o"), snq=V(pre + "self_attn.norm_q.weight"),
                snk=V(pre + "self_attn.norm_k.weight"),
                cq=P_(pre + "cross_attn.q"), ck=P_(pre + "cross_attn.k"), cv=P_(pre + "cross_attn.v"),
                co=P_(pre + "cross_attn.o"), cnq=V(pre + "cross_attn.norm_q.weight"),
                cnk=V(pre + "cross_attn.norm_k.weight"),
                n3_scale=V(pre + "norm3.weight") - 1.0, n3_shift=V(pre + "norm3.bias"),
                f0=P_(pre + "ffn.0"), f2=P_(pre + "ffn.2")))
        # image-to-video models: CLIP-feature MLP and a second key/value projection per block (wan_dit.py:131-134,297)
        self.has_image = "img_emb.proj.1.weight" in sd
        if self.has_image:
            self.img_ln0 = (V("img_emb.proj.0.bias"), V("img_emb.proj.0.weight") - 1.0)   # affine LN as shift, scale
            self.img1, self.img3 = P_("img_emb.proj.1"), P_("img_emb.proj.3")
            self.img_ln4 = (V("img_emb.proj.4.bias"), V("img_emb.proj.4.weight") - 1.0)
            for i, blk in enumerate(self.blocks):
                pre = f"blocks.{i}.cross_attn."
                blk.update(ck_img=P_(pre + "k_img"), cv_img=P_(pre + "v_img"), cnk_img=V(pre + "norm_k_img.weight"))
        if self.P == 1:
            for blk in self.blocks:
                blk["sqkv"] = _stack_linears([blk.pop("sq"), blk.pop("sk"), blk.pop("sv")])   # one N = 3d projection
        self.mod = (torch.stack(mods).contiguous() if mods                  # [L, 6, d]
                    else torch.zeros(0, 6, self.d, dtype=torch.float32, device=self.dev))
        self.head = P_("head.head")
        self.head_mod = V("head.modulation").reshape(2, self.d)
        self.out_dim = self.head.out_features // 4
        self._bufs = None
        self._comm = torch.cuda.Stream(self.dev) if self.overlap else None

    # ------------------------------------------------------------------ buffers
    def prepare(self, frames: int, height: int, width: int, ctx_len: int = 512, text_dim: int = 4096):
        """Buffers for latents [1, C, frames, height, width]; this rank's token slice and RoPE rows."""
        d, dev, P = self.d, self.dev, self.P
        gh, gw = height // 2, width // 2
        S = frames * gh * gw
        Sl = (S + P - 1) // P            # a token count that does not split evenly is padded; the padded rows are
        if self.exchange != "nccl":      # ordinary rows whose results are dropped and that never act as keys
            Sl = (Sl + 127) // 128 * 128                  # the attention kernel reads whole 128-row query tiles per rank
        S_pad = Sl * P
        ffn = self.blocks[0]["f0"].out_features if self.blocks else 4 * d
        qdt = {ops.FMT_BF16: torch.bfloat16, ops.FMT_E4M3: torch.float8_e4m3fn, ops.FMT_INT8: torch.int8}[self.afmt]
        bf, f32 = torch.bfloat16, torch.float32
        C = d // P
        b = dict(S=S, S_pad=S_pad, Sl=Sl, grid=(frames, gh, gw), ctx_len=ctx_len, in_ch=self.patch.in_features // 4)
        b["rope"] = wan_rope_table(frames, gh, gw, device=dev)
        if S_pad > S:   # identity rotation for the padded rows
            pad = torch.zeros(S_pad - S, 64, 2, dtype=b["rope"].dtype, device=dev)
            pad[..., 0] = 1.0
            b["rope"] = torch.cat([b["rope"], pad]).contiguous()
        b["latents"] = torch.zeros(1, b["in_ch"], frames, height, width, dtype=bf, device=dev)
        b["context_in"] = torch.zeros(ctx_len, text_dim, dtype=bf, device=dev)
        b["t"] = torch.zeros(1, dtype=f32, device=dev)
        b["sin"] = torch.zeros(1, self.freq_dim, dtype=f32, device=dev)
        b["th"], b["tvec"] = torch.zeros(d, dtype=f32, device=dev), torch.zeros(d, dtype=f32, device=dev)
        b["tmod"] = torch.zeros(6 * d, dtype=f32, device=dev)
        b["modall"] = torch.zeros(self.L, 6, d, dtype=f32, device=dev)
        b["headmod"] = torch.zeros(2, d, dtype=f32, device=dev)
        b["patches"] = torch.zeros(Sl, self.patch.in_features, dtype=bf, device=dev)
        b["x"] = torch.zeros(Sl, d, dtype=bf, device=dev)
        b["xq"] = torch.zeros(Sl, d if self.afmt == ops.FMT_E4M3 else max(d, ffn), dtype=qdt, device=dev)
        b["rs"] = torch.zeros(max(Sl, ctx_len, IMG_TOKENS), dtype=f32, device=dev)
        b["qkv"] = torch.zeros(Sl, 3 * d, dtype=bf, device=dev)              # fused q | k | v projection of the slice
        b["proj"] = torch.zeros(2, Sl, d, dtype=bf, device=dev)              # cross-attention q and attention output
        b["send"] = torch.zeros(3, P, Sl, C, dtype=bf, device=dev) if P > 1 else None
        b["recv"] = torch.zeros(3, P, Sl, C, dtype=bf, device=dev) if P > 1 else None
        b["ao"] = torch.zeros(P, Sl, C, dtype=bf, device=dev)                # attention out: [S, H/P*128]
        b["ao_back"] = torch.zeros(P, Sl, C, dtype=bf, device=dev) if P > 1 else None
        b["peer"] = None
        if self.exchange != "nccl":
            # this rank's normalised queries [Sl, d] and its returned attention rows [P][Sl][C] live in a buffer every
            # rank maps; flags for the rank barrier behind them
            part = Sl * d * 2
            try:
                pm = PeerMemory(2 * part + 1024, dev, self._group)
            except Exception as e:       # no peer mapping on this system: every tensor goes through the all-to-all
                if self.exchange == "peer":
                    raise
                import sys
                print(f"[wan] peer memory unavailable ({type(e).__name__}: {str(e)[:200]}); using all-to-all", file=sys.stderr)
                pm = None
            # the ranks must agree (a rank that fell back while another did not would wait for ever)
            ok = torch.tensor([1 if pm is not None else 0], dtype=torch.int32, device=dev)
            self.xchg.dist.all_reduce(ok, op=self.xchg.dist.ReduceOp.MIN, group=self._group)
            if int(ok.item()) == 0:
                if self.exchange == "peer":
                    raise RuntimeError("peer memory could not be mapped on every rank")
                self.exchange = "nccl"
                return self.prepare(frames, height, width, ctx_len, text_dim)
            self.exchange = "peer"
            b["peer"] = pm
            b["qn"] = pm.local[:part].view(bf).view(Sl, d)
            b["ao_back"] = pm.local[part:2 * part].view(bf).view(P, Sl, C)
            b["flags"] = [ptr + 2 * part for ptr in pm.ptrs]
            # peer r's queries of this rank's head group; this rank's chunk of peer r's returned attention rows
            b["attn_ws"] = ops.flash_attn_workspace(dev) if self.tail_split else None
            b["q_parts"] = [ptr + self.rank * C * 2 for ptr in pm.ptrs]
            b["o_parts"] = [ptr + part + self.rank * Sl * C * 2 for ptr in pm.ptrs]
            self.xchg.dist.barrier(group=self._group)           # every rank's flags are zero before the first signal
        # FFN hidden: bf16 (then row-quantised into xq) - or, with FP8 weights, e4m3 written by the first FFN GEMM itself
        # (its own buffer: that GEMM still reads its operand from xq)
        b["hid"] = torch.zeros(Sl, ffn, dtype=qdt if self.afmt == ops.FMT_E4M3 else bf, device=dev)
        # context rows: [CLIP tokens (image-to-video only) | text tokens], as the reference concatenates them
        n_img = IMG_TOKENS if self.has_image else 0
        L_all = n_img + ctx_len
        b["n_img"] = n_img
        b["ctx"] = torch.zeros(L_all, d, dtype=bf, device=dev)
        b["ctx_h"] = torch.zeros(max(ctx_len, n_img), max(d, 1280 if n_img else 0), dtype=bf, device=dev)
        b["ctxq"] = torch.zeros(L_all, max(d, text_dim, 1280 if n_img else 0), dtype=qdt, device=dev)
        b["ctx_rs"] = torch.zeros(L_all, dtype=f32, device=dev)
        # cross-attention keys and values of every block: they depend on the context only (wan_dit.py:143-149 applied to
        # the output of text_embedding), so they are computed once per prompt and reused by every later step
        b["ckv"] = torch.zeros(max(self.L, 1), 2, L_all, d, dtype=bf, device=dev)
        b["ctx_key"] = None
        if n_img:
            b["clip_in"] = torch.zeros(n_img, 1280, dtype=bf, device=dev)
        b["out_tok"] = torch.zeros(Sl, self.head.out_features, dtype=bf, device=dev)
        b["out_all"] = torch.zeros(S_pad, self.head.out_features, dtype=bf, device=dev) if P > 1 else None
        b["out_lat"] = torch.zeros(1, self.out_dim, frames, height, width, dtype=bf, device=dev)
        self._bufs = b
        return self

    # -------------------------------------------------------------------- pieces
    def _gemv(self, p: PackedLinear, x, out, **kw):
        ops.gemv(p.w, x, p.scale, p.bias, out=out, **kw)

    def _quant(self, x, out, rs):
        if self.afmt == ops.FMT_BF16:
            return x, None
        ops.quant_rows(x, self.afmt, out=out, row_scale=rs)
        return out, rs

    def _ln(self, x, shift, scale, out, rs):
        y, s = ops.ln_modulate(x, shift, scale, self.eps, self.afmt, out=out, row_scale=rs)
        return y, (s if self.afmt != ops.FMT_BF16 else None)

    def _gemm(self, a, rs, p: PackedLinear, **kw):
        return ops.gemm(a, p.w, row_scale=rs, col_scale=p.scale, bias=p.bias, **kw)

    def set_inputs(self, x, context, timestep, clip_feature=None, y=None):
        b = self._bufs
        if self.has_image:
            if clip_feature is None or y is None:
                raise ValueError("an image-to-video model needs clip_feature and y")
            nx = x.shape[1]
            b["latents"][:, :nx].copy_(x, non_blocking=True)          # torch.cat([x, y], dim=1), wan_dit.py:331
            b["latents"][:, nx:].copy_(y, non_blocking=True)
            b["clip_in"].copy_(clip_feature.reshape(b["clip_in"].shape), non_blocking=True)
        else:
            if clip_feature is not None or y is not None:
                raise ValueError("this model has no image branch (no img_emb / k_img / v_img weights)")
            b["latents"].copy_(x.reshape(b["latents"].shape), non_blocking=True)
        # the cross-attention keys / values are cached per context: the same memory, unmodified since the last call (a
        # pipeline passes its prompt embedding again at every denoising step), keeps them.  The tensors are held meanwhile,
        # so that no other prompt's embedding can be put where a dropped one lay.
        key = (context.data_ptr(), context._version, tuple(context.shape), context.stride(), context.dtype, str(context.device),
               None if clip_feature is None else (clip_feature.data_ptr(), clip_feature._version))
        if b.get("ctx_key") != key:
            b["ctx_key"], b["ctx_valid"], b["ctx_held"] = key, False, (context, clip_feature)
            b["context_in"].copy_(context.reshape(b["context_in"].shape), non_blocking=True)
        b["t"].copy_(timestep.reshape(1), non_blocking=True)

    def _exchange(self, send, recv, after_event=None):
        """all-to-all on the communication stream (when overlapping) once the producing kernel has finished;
        returns an event the consumer waits on."""
        if not self.overlap:
            self.xchg(send, recv)
            return None
        cur = torch.cuda.current_stream(self.dev)
        ready = torch.cuda.Event()
        ready.record(cur)
        with torch.cuda.stream(self._comm):
            self._comm.wait_event(ready)
            self.xchg(send, recv)
            done = torch.cuda.Event()
            done.record(self._comm)
        return done

    def _barrier(self):
        """All ranks of the group, on the current stream (``dsb_rank_barrier`` over the mapped flag arrays)."""
        self._epoch += 1
        ops.rank_barrier(self._bufs["flags"], self.rank, self._epoch)

    def step(self):
        b, d, H, P = self._bufs, self.d, self.H, self.P
        Sl, S, Hl, C = b["Sl"], b["S"], self.H // self.P, self.d // self.P
        x, xq, rs = b["x"], b["xq"], b["rs"]
        xq_d = xq[:, :d]
        row0 = self.rank * Sl
        cur = torch.cuda.current_stream(self.dev)
        # time embedding / projection (wan_dit.py:327-328); the reference casts the fp64 sinusoid to the model dtype
        ops.timestep_embedding(b["t"], self.freq_dim, 1.0, 1, round_bf16=True, out=b["sin"])
        self._gemv(self.time0, b["sin"][0], b["th"], act_out=ops.ACT_SILU)
        self._gemv(self.time2, b["th"], b["tvec"])
        self._gemv(self.tproj, b["tvec"], b["tmod"], act_in=ops.ACT_SILU)
        torch.add(self.mod, b["tmod"].view(1, 6, d), out=b["modall"])          # (modulation + t_mod), every block
        torch.add(self.head_mod, b["tvec"].view(1, d), out=b["headmod"])       # wan_dit.py:235
        tdim = b["context_in"].shape[1]
        n_img, L = b["n_img"], b["ctx_len"]
        txt_rows = slice(n_img, n_img + L)
        ckv = b["ckv"]
        if not b.get("ctx_valid", False):
            # text embedding (wan_dit.py:329) and every block's cross-attention keys / values (:143-149): functions of
            # the context alone, replicated on every rank, computed on the first step after the context changed
            ctxq_t, crs_t, ctx_h = b["ctxq"][txt_rows], b["ctx_rs"][txt_rows], b["ctx_h"]
            a, s = self._quant(b["context_in"], ctxq_t[:, :tdim], crs_t)
            self._gemm(a, s, self.text0, act=ops.ACT_GELU_TANH, out=ctx_h[:L, :d])
            a, s = self._quant(ctx_h[:L, :d], ctxq_t[:, :d], crs_t)
            self._gemm(a, s, self.text2, out=b["ctx"][txt_rows])
            if n_img:   # CLIP tokens through img_emb (LN -> Linear -> GELU -> Linear -> LN, wan_dit.py:196-216), eps 1e-5
                ctxq_i, crs_i = b["ctxq"][:n_img], b["ctx_rs"][:n_img]
                a, s = ops.ln_modulate(b["clip_in"], self.img_ln0[0], self.img_ln0[1], 1e-5, self.afmt,
                                       out=ctxq_i[:, :1280], row_scale=crs_i)
                s = s if self.afmt != ops.FMT_BF16 else None
                self._gemm(a, s, self.img1, act=ops.ACT_GELU, out=ctx_h[:n_img, :1280])
                a, s = self._quant(ctx_h[:n_img, :1280], ctxq_i[:, :1280], crs_i)
                tmp = ckv[0, 0, :n_img]                                        # free until the loop below fills it
                self._gemm(a, s, self.img3, out=tmp)
                ops.ln_modulate(tmp, self.img_ln4[0], self.img_ln4[1], 1e-5, ops.FMT_BF16, out=b["ctx"][:n_img])
            cq_, cs_ = self._quant(b["ctx"], b["ctxq"][:, :d], b["ctx_rs"])    # quantised context, shared by all blocks
            cq_t, cs_t = cq_[txt_rows], (None if cs_ is None else cs_[txt_rows])
            for li, blk in enumerate(self.blocks):
                ck_t, cv_t = ckv[li, 0, txt_rows], ckv[li, 1, txt_rows]
                self._gemm(cq_t, cs_t, blk["ck"], out=ck_t)
                ops.rmsnorm_full(ck_t, blk["cnk"], None, 0, self.eps)
                self._gemm(cq_t, cs_t, blk["cv"], out=cv_t)
                if n_img:
                    cq_i, cs_i = cq_[:n_img], (None if cs_ is None else cs_[:n_img])
                    ck_i, cv_i = ckv[li, 0, :n_img], ckv[li, 1, :n_img]
                    self._gemm(cq_i, cs_i, blk["ck_img"], out=ck_i)
                    ops.rmsnorm_full(ck_i, blk["cnk_img"], None, 0, self.eps)
                    self._gemm(cq_i, cs_i, blk["cv_img"], out=cv_i)
            b["ctx_valid"] = True
        # patch embedding: Conv3d with kernel = stride = (1,2,2) is a Linear over (c, y, z) patches (wan_dit.py:271-273)
        fr, gh, gw = b["grid"]
        Cin = b["in_ch"]
        # dsb_patchify gathers this rank's token rows straight from the latents and quantises them in the same pass
        # (rows past the last token of a padded sequence come out as zeros)
        if self.afmt == ops.FMT_BF16:
            a, s = ops.patchify(b["latents"], row0, Sl, ops.FMT_BF16, out=b["patches"])
        else:
            a, s = ops.patchify(b["latents"], row0, Sl, self.afmt, out=xq[:, :Cin * 4], row_scale=rs[:Sl])
        self._gemm(a, s, self.patch, out=x)

        rope = b["rope"]
        proj, qkv = b["proj"], b["qkv"]
        ao = b["ao"]
        q_s, k_s, v_s = qkv[:, :d], qkv[:, d:2 * d], qkv[:, 2 * d:]          # column blocks of the fused projection
        for li, blk in enumerate(self.blocks):
            m = b["modall"][li]
            # ---- self-attention (wan_dit.py:101-107) with the head exchange around it: q, k and v in ONE GEMM
            a, sc = self._ln(x, m[0], m[1], xq_d, rs[:Sl])
            if P == 1:
                self._gemm(a, sc, blk["sqkv"], out=qkv)
                ops.rmsnorm_full(q_s, blk["snq"], rope, row0, self.eps)
                ops.rmsnorm_full(k_s, blk["snk"], rope, row0, self.eps)
                q4, k4, v4 = (t.unflatten(1, (H, 128)).unsqueeze(0) for t in (q_s, k_s, v_s))
                ops.flash_attn(q4, k4, v4, out=ao.view(1, S, H, 128))
                att3 = None
            else:
                send, recv = b["send"], b["recv"]
                S_pad = b["S_pad"]
                peer = self.exchange == "peer"
                # k, v, q are projected one after the other so that each tensor leaves for its head group's rank
                # under the projection of the next one
                self._gemm(a, sc, blk["sk"], out=k_s)
                ops.rmsnorm_full(k_s, blk["snk"], rope, row0, self.eps, out=send[1], chunks=P)
                e1 = self._exchange(send[1], recv[1])
                self._gemm(a, sc, blk["sv"], out=v_s)
                send[2].copy_(v_s.unflatten(1, (P, C)).permute(1, 0, 2))
                e2 = self._exchange(send[2], recv[2])
                self._gemm(a, sc, blk["sq"], out=q_s)
                if peer:
                    # the queries stay where they are: every rank's attention kernel fetches the rows it needs
                    ops.rmsnorm_full(q_s, blk["snq"], rope, row0, self.eps, out=b["qn"])
                    self._barrier()                                   # every rank's queries are written
                    e0 = None
                else:
                    ops.rmsnorm_full(q_s, blk["snq"], rope, row0, self.eps, out=send[0], chunks=P)
                    e0 = self._exchange(send[0], recv[0])
                for e in (e0, e1, e2):
                    if e is not None:
                        cur.wait_event(e)
                k4, v4 = (recv[i].view(S_pad, Hl, 128)[:S].unsqueeze(0) for i in (1, 2))   # real tokens only as keys
                if peer:
                    ops.flash_attn_parts(b["q_parts"], Sl, (d, 128), k4, v4, b["o_parts"], Sl, (C, 128), Hl, S_pad,
                                         workspace=b["attn_ws"])
                    self._barrier()                                   # every rank's output rows have arrived
                else:
                    q4 = recv[0].view(1, S_pad, Hl, 128)
                    ops.flash_attn(q4, k4, v4, out=ao.view(1, S_pad, Hl, 128))
                    e3 = self._exchange(ao, b["ao_back"])
                    if e3 is not None:
                        cur.wait_event(e3)
                att3 = b["ao_back"]
            if self.afmt == ops.FMT_BF16:
                att = ao.view(S, d) if P == 1 else att3.permute(1, 0, 2).reshape(Sl, d)
                a, sc = att, None
            elif P == 1:
                a, sc = self._quant(ao.view(S, d), xq_d, rs[:Sl])
            else:
                a, sc = ops.quant_rows_chunked(att3, self.afmt, out=xq_d, row_scale=rs[:Sl])
            self._gemm(a, sc, blk["so"], gate=m[2], resid=x, out=x)
            # ---- cross-attention (wan_dit.py:136-152): no exchange, the context is replicated
            a, sc = self._ln(x, blk["n3_shift"], blk["n3_scale"], xq_d, rs[:Sl])
            self._gemm(a, sc, blk["cq"], out=proj[0])
            ops.rmsnorm_full(proj[0], blk["cnq"], None, 0, self.eps)
            ck_t, cv_t = ckv[li, 0, txt_rows], ckv[li, 1, txt_rows]
            ops.flash_attn(proj[0].view(1, Sl, H, 128), ck_t.view(1, L, H, 128), cv_t.view(1, L, H, 128),
                           out=proj[1].view(1, Sl, H, 128))
            if n_img:   # the CLIP tokens have their own k/v projection; the two attention outputs add (wan_dit.py:147-151)
                ck_i, cv_i = ckv[li, 0, :n_img], ckv[li, 1, :n_img]
                att_i = qkv[:, :d]                                             # free until the next block's projection
                ops.flash_attn(proj[0].view(1, Sl, H, 128), ck_i.view(1, n_img, H, 128), cv_i.view(1, n_img, H, 128),
                               out=att_i.unflatten(1, (H, 128)).unsqueeze(0))
                ops.gate_residual(proj[1], att_i, None, out=proj[1])           # bf16(x + y)
            a, sc = self._quant(proj[1], xq_d, rs[:Sl])
            self._gemm(a, sc, blk["co"], resid=x, out=x)
            # ---- FFN (wan_dit.py:179-182,191-192)
            a, sc = self._ln(x, m[3], m[4], xq_d, rs[:Sl])
            if self.afmt == ops.FMT_E4M3:
                # GELU(hidden) leaves the GEMM as e4m3 with unit scale (the reference's own activation rule,
                # utils/fp8_linear.py:35): no row quantiser in front of the second FFN Linear
                hq = b["hid"]
                p0 = blk["f0"]
                ops.gemm_group([dict(a=a, w=p0.w, row_scale=sc, col_scale=p0.scale, bias=p0.bias,
                                     act=ops.ACT_GELU_TANH, out=hq)])
                a, sc = hq, None
            else:
                self._gemm(a, sc, blk["f0"], act=ops.ACT_GELU_TANH, out=b["hid"])
                a, sc = self._quant(b["hid"], xq[:, :b["hid"].shape[1]], rs[:Sl])
            self._gemm(a, sc, blk["f2"], gate=m[5], resid=x, out=x)
        # ---- head (wan_dit.py:234-237) and unpatchify (:307-317)
        hm = b["headmod"]
        a, sc = self._ln(x, hm[0], hm[1], xq_d, rs[:Sl])
        self._gemm(a, sc, self.head, out=b["out_tok"])
        if P > 1:
            self.xchg.dist.all_gather_into_tensor(b["out_all"], b["out_tok"], group=self.xchg.group)
            tok = b["out_all"][:S]
        else:
            tok = b["out_tok"]
        return ops.unpatchify(tok, self.out_dim, fr, gh, gw, True, out=b["out_lat"])

    def forward(self, x, context, timestep, clip_feature=None, y=None):
        """Signature of ``WanDiT.forward`` (wan_dit.py:319-326).  ``clip_feature`` [1,257,1280] and ``y`` (conditioning
        latents on the grid of ``x``) are required by image-to-video weights and rejected by text-to-video ones."""
        if x.shape[0] != 1 or context.shape[0] != 1:
            raise ValueError("WanDiTEngine runs one sample per call (batch 1); split a CFG batch into two calls or use "
                             "UlyssesParallelModel(batch_parallelism=2)")
        b = self._bufs
        shape = (x.shape[2], x.shape[3], x.shape[4], context.shape[1], context.shape[2])
        if b is None or (b["latents"].shape[2], b["latents"].shape[3], b["latents"].shape[4], b["ctx_len"],
                         b["context_in"].shape[1]) != shape:
            self.prepare(*shape)
        self.set_inputs(x, context, timestep, clip_feature, y)
        return self.step().clone()

    __call__ = forward

    def hidden(self):
        """This rank's slice of the hidden state after the last block (for tests)."""
        return self._bufs["x"]
