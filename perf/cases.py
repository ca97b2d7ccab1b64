"""The work that users of this package have it do, as measurable cases.

A case is one call of a public entry point on a KV cache of one shape:

    call      decode, decode_many, decode_many_host, from_bytes_many     retrieval of a stored cache
              encode, encode_many, encode_levels                         storing one
              round_trip                                                 a chunk to bytes and back
              torchac                                                    the extension module's entry points on symbols
    layers, heads, head, tokens    the KV cache; 32 layers use the 7B bin settings, any other number the first
                                   layers of the 70B settings (layer sharding)
    chunk     tokens of one serializer call
    dtype     float16 or bfloat16, of the KV that goes in and comes out
    fmt       "vllm" [L, 2, T, H, D] or "huggingface" [L, 2, H, T, D]
    wire      "pickle" (the reference's blob) or "flat" (the CGB2 container)
    bins      "default", "half", "quarter", or a level "1", "2", "3" of the Mistral settings
    rho       token-to-token correlation of the keys

KV comes from the package's synthetic generator (AR(1) series per channel, lognormal channel scales, 2 % of the
key channels ten times larger).
"""
import math

import torch

from cachegen_b200 import synth, torchac_cuda
from cachegen_b200.config import LMCacheEngineConfig, LMCacheEngineMetadata
from cachegen_b200.serde import CacheGenConfig, CacheGenDeserializer, CacheGenGPUBytestream, CacheGenSerializer
from cachegen_b200.serde import cachegen_basics, cachegen_decoder, cachegen_encoder

_DTYPES = {"float16": torch.float16, "bfloat16": torch.bfloat16}
_LEVELS = {"1": (16, 16, 12, 16, 12), "2": (32, 16, 16, 32, 16), "3": (32, 32, 32, 32, 32)}
_DIVISOR = {"default": 1, "half": 2, "quarter": 4}


def _case(name, call, layers, heads, head, tokens, chunk=256, dtype="float16", fmt="vllm", wire="pickle",
          bins="default", rho=0.9):
    return {"name": name, "call": call, "layers": layers, "heads": heads, "head": head, "tokens": tokens,
            "chunk": chunk, "dtype": dtype, "fmt": fmt, "wire": wire, "bins": bins, "rho": rho}


def listed():
    return [
        # the ragged end of a request's cache: a few tokens, already on the GPU, where launches and host work count
        _case("decode_tail_37", "decode", 32, 8, 128, 37, dtype="bfloat16"),
        # the same end to a remote store and back, on one of eight layer shards: one small container as bytes
        _case("round_trip_tail_61", "round_trip", 10, 8, 128, 61, dtype="bfloat16", wire="flat"),
        # what a cache engine does for every 256 tokens it stores on the GPU
        _case("encode_chunk_256", "encode", 32, 32, 128, 256),
        # a whole context in one serializer call, as evaluation scripts make it, in the transposed layout
        _case("encode_context_1999", "encode", 32, 8, 128, 1999, chunk=1999, fmt="huggingface", bins="half"),
        # one chunk to a remote store and back in the reference's blob format
        _case("round_trip_256", "round_trip", 32, 32, 128, 256),
        # a 1,024-token request fetched from a remote store: four blobs in host memory to one KV blob
        _case("from_bytes_many_1024", "from_bytes_many", 32, 32, 128, 1024),
        # a long prompt's cache stored chunk after chunk
        _case("encode_many_3072", "encode_many", 32, 32, 128, 3072),
        # a chunk at the three quality levels that adaptive streaming chooses from
        _case("encode_levels_256", "encode_levels", 32, 8, 128, 256, dtype="bfloat16", bins="2"),
        # a long context loaded from chunks in GPU memory: multi-head shape
        _case("decode_many_8192", "decode_many", 32, 32, 128, 8192),
        # the same for grouped-query heads, a longer context and the finest level
        _case("decode_many_32768_gqa", "decode_many", 32, 8, 128, 32768, dtype="bfloat16", bins="3", rho=0.95),
        # a large model's context loaded from containers in pinned host memory
        _case("decode_host_4096_70b", "decode_many_host", 80, 8, 128, 4096, wire="flat"),
        # code written against the extension module: tables, streams and symbols of one chunk
        _case("torchac_256", "torchac", 32, 32, 128, 256),
    ]


# the most KV values (layers * 2 * tokens * channels) of a drawn case and the most chunks of a call
_MOST = {"decode": 32 * 2 * 256 * 4096, "encode": 32 * 2 * 1999 * 1024,
         "round_trip": 32 * 2 * 256 * 4096, "from_bytes_many": 32 * 2 * 1024 * 4096, "encode_many": 32 * 2 * 3072 * 4096,
         "encode_levels": 32 * 2 * 256 * 1024, "decode_many": 32 * 2 * 8192 * 4096, "decode_many_host": 80 * 2 * 4096 * 1024,
         "torchac": 32 * 2 * 256 * 4096}
_ONE_CHUNK = ("decode", "round_trip", "encode_levels", "torchac")


def draw(rng):
    call = rng.choice(sorted(_MOST))
    layers, heads, head = rng.choice([(32, 32, 128), (32, 8, 128), (80, 8, 128), (40, 8, 128), (10, 8, 128),
                                      (32, rng.randint(1, 16), rng.choice([64, 80, 96, 112, 128, 256]))])
    most = max(1, _MOST[call] // (layers * 2 * heads * head))
    if call in _ONE_CHUNK:
        most = min(most, 256)
    elif call == "encode":
        most = min(most, 2048)
    elif call == "encode_many":
        most = min(most, 12 * 256)
    else:
        most = min(most, 32768)
    tokens = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    chunk = tokens if call == "encode" else max(tokens, 256) if call in _ONE_CHUNK else 256
    wire = "flat" if call == "decode_many_host" else "pickle"
    if call in ("round_trip", "from_bytes_many"):
        wire = rng.choice(["pickle", "flat"])
    bins = "2" if call == "encode_levels" else rng.choice(["default", "half", "quarter", "1", "3"])
    case = _case("", call, layers, heads, head, tokens, chunk, rng.choice(sorted(_DTYPES)),
                 rng.choice(["vllm", "huggingface"]), wire, bins, rng.choice([0.9, 0.95]))
    del case["name"]
    return case


def _config(layers, bins):
    model = "lmsys/longchat-7b-16k" if layers == 32 else "Yukang/LongAlpaca-70B-16k"
    config = CacheGenConfig.from_model_name(model)
    if bins in _LEVELS:
        k1, k2, k3, v1, v2 = _LEVELS[bins]
        config = CacheGenConfig(config.key_first_layers, config.key_second_layers, config.key_third_layers, k1, k2, k3,
                                config.value_first_layers, v1, v2)
    elif _DIVISOR[bins] > 1:
        config = config.with_bins_divided(_DIVISOR[bins])
    whole = config.max_bins
    return (config if layers == config.num_layers else config.layer_slice(0, layers)), whole


def _slot(values, streams):
    """Room in a store's pool for the streams of one chunk: the finest level needs five bits a value."""
    return torch.zeros(values * 3 // 4 + 4 * streams, dtype=torch.uint8, device="cuda")


def _put(chunk, slot):
    """An encoded chunk in its place: the streams, whose size differs from chunk to chunk, in the slot."""
    out, at = [chunk.cdf, chunk.max_tensors_key, chunk.max_tensors_value, slot], 0
    for piece in chunk.data_chunks:
        n = piece.bytestream.numel()
        slot[at:at + n].copy_(piece.bytestream)
        at += n
        out.append(piece.bytestream_lengths)
    return out


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.call = case["call"]
    dtype = _DTYPES[case["dtype"]]
    config, table_max_bins = _config(case["layers"], case["bins"])
    engine = LMCacheEngineConfig.from_defaults(chunk_size=max(case["chunk"], min(case["tokens"], 256)))
    meta = LMCacheEngineMetadata("cases", 1, 0, case["fmt"])
    s.serializer = CacheGenSerializer(engine, meta, config, case["wire"], table_max_bins)
    s.deserializer = CacheGenDeserializer(engine, meta, config, out_dtype=dtype)
    kv = synth.generate_kv(case["layers"], case["heads"], case["head"], case["tokens"], seed, key_rho=case["rho"],
                           device="cuda", dtype=dtype)
    if case["fmt"] == "huggingface":
        kv = kv.permute(0, 1, 3, 2, 4).contiguous()
    L, T, C = case["layers"], case["tokens"], case["heads"] * case["head"]
    axis = 2 if case["fmt"] == "vllm" else 3
    parts = kv.split(case["chunk"], dim=axis)
    if s.call in ("encode", "encode_many", "encode_levels", "round_trip"):
        s.kv, s.chunk = kv, case["chunk"]
        if s.call == "encode_levels":
            s.levels = [_config(L, level)[0] for level in ("1", "2", "3")]
        if s.call != "round_trip":
            s.slots = [_slot(p.numel(), -(-p.shape[axis] // 256) * 2 * L * C)
                       for p in (parts * 3 if s.call == "encode_levels" else parts)]
        return s
    if s.call in ("decode", "decode_many"):
        s.chunks = [s.serializer.encode(p) for p in parts]
    elif s.call == "decode_many_host":
        s.chunks = [s.serializer.encode_flat(p).pin_memory() for p in parts]
    elif s.call == "from_bytes_many":
        s.blobs = [s.serializer.to_bytes(p) for p in parts]
    else:  # torchac: what its callers hold is symbols, and buffers of the shapes that the coder fills
        bins = torch.cat((s.serializer.key_bins, s.serializer.value_bins))
        x = kv if case["fmt"] == "vllm" else kv.permute(0, 1, 3, 2, 4)
        x = x.transpose(0, 1).reshape(2 * L, T, C)
        s.symbols, s.max_bins = cachegen_encoder.torch_quant_vectorized(bins, x)[0], table_max_bins
        s.buffer = torch.empty((2 * L, C, 520), dtype=torch.uint8, device=x.device)
        s.lengths = torch.empty((2 * L, C), dtype=torch.int32, device=x.device)
        s.slots = [_slot(x.numel(), 2 * L * C)]
        s.decoded = torch.empty((2 * L, T, C), dtype=torch.uint8, device=x.device)
    return s


def run(s):
    if s.call == "decode":
        return s.deserializer.decode(s.chunks[0])
    if s.call == "decode_many":
        return s.deserializer.decode_many(s.chunks)
    if s.call == "decode_many_host":
        return s.deserializer.decode_many_host(s.chunks)
    if s.call == "from_bytes_many":
        return s.deserializer.from_bytes_many(s.blobs)
    if s.call == "encode":
        return _put(s.serializer.encode(s.kv), s.slots[0])
    if s.call == "encode_many":
        return [_put(c, slot) for c, slot in zip(s.serializer.encode_many(s.kv, s.chunk), s.slots)]
    if s.call == "encode_levels":
        return [_put(c, slot) for c, slot in zip(s.serializer.encode_levels(s.kv, s.levels), s.slots)]
    if s.call == "round_trip":
        # the bytes differ in length from cache to cache, so what comes back from them is the output
        return s.deserializer.from_bytes(s.serializer.to_bytes(s.kv))
    cdf = torchac_cuda.calculate_cdf(s.symbols, s.max_bins)
    streams = cachegen_encoder.encode_ntokens(cdf, s.symbols, s.buffer, s.lengths)
    cachegen_decoder.decode_chunk(cdf, CacheGenGPUBytestream(streams, s.lengths, s.symbols.shape[1]), s.decoded)
    slot = s.slots[0]
    slot[:streams.numel()].copy_(streams)
    return cdf, slot, s.lengths, s.decoded


def _stream_bits(config, layers):
    """Bits of one token and channel of every row, roughly: a value costs log2(bins / 2 - 1) less a third of a
    bit at these distributions, a key two and a half bits less than that."""
    key = cachegen_basics.make_key_bins(config, "cpu").tolist()
    value = cachegen_basics.make_value_bins(config, "cpu").tolist()
    one = lambda b, less: max(0.3, math.log2(max(1.0, b // 2 - 1)) - less)
    return sum(one(b, 2.8) for b in key) + sum(one(b, 0.3) for b in value)


def work(case):
    L, C, T = case["layers"], case["heads"] * case["head"], case["tokens"]
    config, lp = _config(L, case["bins"])
    lp += 1
    kv = 2 * L * T * C * 2
    chunks = -(-T // case["chunk"])
    subs = sum(-(-min(case["chunk"], T - s) // 256) for s in range(0, T, case["chunk"]))
    streams = _stream_bits(config, L) / 8 * C * T
    tables = chunks * 2 * L * C * (lp * 2 if case["wire"] == "pickle" else 8)
    lengths = subs * 2 * L * C * (4 if case["wire"] == "pickle" else 2)
    coded = int(streams + tables + lengths + 2 * L * T * 2)
    values = 2 * L * T * C
    if case["call"] == "torchac":  # symbols in, symbols out, and the streams both ways
        return {"bytes": 2 * values + 2 * coded, "flops": 0}
    if case["call"] == "round_trip":
        return {"bytes": 2 * kv + 2 * coded, "flops": 4 * values}
    if case["call"] == "encode_levels":
        return {"bytes": kv + 3 * coded, "flops": 9 * values}
    return {"bytes": kv + coded, "flops": values * (1 if case["call"].startswith(("decode", "from")) else 3)}


def tolerance(case):
    # streams, tables and symbols are whole numbers; a decoded value is one product in fp32 and one rounding
    return "exact"
