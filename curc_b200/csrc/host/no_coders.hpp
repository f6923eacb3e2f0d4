// Stand-in for the vendored stream coders' headers, for a build where the
// reference's source tree is not present (CURC_NO_CODERS): the device path,
// ingest and the other host code build and run as usual, and every call that
// would code or decode a stream throws.  Names and signatures only.
#pragma once
#include <cstddef>
#include <cstdint>
#include <istream>
#include <ostream>
#include <stdexcept>
#include <string>

namespace no_coders {
[[noreturn]] inline void fail() {
    throw std::runtime_error("built without the reference's stream coders");
}
}  // namespace no_coders

using Byte = unsigned char;
using SizeT = size_t;
using SRes = int;
enum { SZ_OK = 0, LZMA_PROPS_SIZE = 5, LZMA_FINISH_ANY = 0 };
enum : uint8_t { LZMA_CODER = 1, PPMD7_CODER = 3, VARLEN_DNA_CODER = 11, COMPOUND_CODER_TYPE = 77 };
enum : unsigned { PPMD7_MIN_ORDER = 2, PPMD7_MAX_ORDER = 64, PPMD7_MIN_MEM_SIZE = 1u << 11, PPMD7_MAX_MEM_SIZE = ~0u - 36 };
constexpr double COMPRESSION_ESTIMATION_UINT8_BITMAP = 1, COMPRESSION_ESTIMATION_MIS_SYM = 1;
inline double simpleUintCompressionEstimate(uint64_t, uint64_t) { no_coders::fail(); }

struct ISzAlloc {};
inline ISzAlloc g_Alloc;
struct IByteOut { void (*Write)(const IByteOut*, Byte); };
struct IByteIn { Byte (*Read)(const IByteIn*); };
struct CPpmd7 {};
struct CPpmd7z_RangeEnc { IByteOut* Stream; };
struct CPpmd7z_RangeDec { struct { } vt; IByteIn* Stream; };
inline void Ppmd7_Construct(CPpmd7*) { no_coders::fail(); }
inline int Ppmd7_Alloc(CPpmd7*, uint32_t, ISzAlloc*) { no_coders::fail(); }
inline void Ppmd7_Init(CPpmd7*, unsigned) { no_coders::fail(); }
inline void Ppmd7_Free(CPpmd7*, ISzAlloc*) { no_coders::fail(); }
inline void Ppmd7z_RangeEnc_Init(CPpmd7z_RangeEnc*) { no_coders::fail(); }
inline void Ppmd7z_RangeEnc_FlushData(CPpmd7z_RangeEnc*) { no_coders::fail(); }
inline void Ppmd7_EncodeSymbol(CPpmd7*, CPpmd7z_RangeEnc*, int) { no_coders::fail(); }
inline void Ppmd7z_RangeDec_CreateVTable(CPpmd7z_RangeDec*) { no_coders::fail(); }
inline int Ppmd7z_RangeDec_Init(CPpmd7z_RangeDec*) { no_coders::fail(); }
inline int Ppmd7z_RangeDec_IsFinishedOK(CPpmd7z_RangeDec*) { no_coders::fail(); }
template <class V>
int Ppmd7_DecodeSymbol(CPpmd7*, V*) { no_coders::fail(); }

struct CLzmaEncProps { int level, lc, lp, pb, fb, numThreads; uint32_t dictSize; uint64_t reduceSize; };
enum ELzmaStatus { LZMA_STATUS_NOT_SPECIFIED };
inline void LzmaEncProps_Init(CLzmaEncProps*) { no_coders::fail(); }
template <class... A>
SRes LzmaEncode(A...) { no_coders::fail(); }
template <class... A>
SRes LzmaDecode(A...) { no_coders::fail(); }

struct FL2_CStream;
struct FL2_DStream;
struct FL2_inBuffer { const void* src; size_t size, pos; };
struct FL2_outBuffer { void* dst; size_t size, pos; };
inline FL2_CStream* FL2_createCStreamMt(unsigned, int) { no_coders::fail(); }
inline size_t FL2_initCStream(FL2_CStream*, int) { no_coders::fail(); }
inline size_t FL2_compressStream(FL2_CStream*, FL2_outBuffer*, FL2_inBuffer*) { no_coders::fail(); }
inline size_t FL2_endStream(FL2_CStream*, FL2_outBuffer*) { no_coders::fail(); }
inline size_t FL2_freeCStream(FL2_CStream*) { no_coders::fail(); }
inline FL2_DStream* FL2_createDStreamMt(unsigned) { no_coders::fail(); }
inline size_t FL2_initDStream(FL2_DStream*) { no_coders::fail(); }
inline size_t FL2_decompressStream(FL2_DStream*, FL2_outBuffer*, FL2_inBuffer*) { no_coders::fail(); }
inline size_t FL2_freeDStream(FL2_DStream*) { no_coders::fail(); }
inline unsigned FL2_isError(size_t) { no_coders::fail(); }
inline const char* FL2_getErrorName(size_t) { no_coders::fail(); }

struct RangeCoder {
    void output(char*) { no_coders::fail(); }
    void input(char*) { no_coders::fail(); }
    void StartEncode() {}
    void StartDecode() {}
    void FinishEncode() {}
    void FinishDecode() {}
    int size_out() { no_coders::fail(); }
};
template <size_t N>
struct SIMPLE_MODEL {
    void encodeSymbol(RangeCoder*, uint16_t) { no_coders::fail(); }
    uint16_t decodeSymbol(RangeCoder*) { no_coders::fail(); }
};

namespace PgSAHelpers {
struct VarLenDNACoder {
    enum : uint8_t { STATIC_CODES_CODER_PARAM = 0, DYNAMIC_CODES_CODER_PARAM = 1, AG_EXTENDED_CODES_ID = 0 };
    static int getCoderParam(int, int) { no_coders::fail(); }
    static int Compress(unsigned char*&, size_t&, const unsigned char*, size_t, int) { no_coders::fail(); }
};
}  // namespace PgSAHelpers
inline char* Compress(size_t&, const char*, size_t, uint8_t, uint8_t, int, double) { no_coders::fail(); }
inline void Uncompress(char*, size_t, const char*, size_t, uint8_t) { no_coders::fail(); }
inline void writeCompressed(std::ostream&, const char*, size_t, uint8_t, uint8_t, int, double) { no_coders::fail(); }
inline void readCompressed(std::istream&, std::string&) { no_coders::fail(); }
namespace lzma2 {
inline void lzma2_compress(const char*, const char*, int, int) { no_coders::fail(); }
inline void lzma2_decompress(const char*, const char*) { no_coders::fail(); }
}  // namespace lzma2
