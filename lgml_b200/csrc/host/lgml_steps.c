/* What a step's description is made of, on the host: token lists to 32-bit integers, positions, tiles of requests, and the keys of full
 * pages.  Called with the interpreter's lock held (the lists are Python's own), so the few functions of its stable interface that are
 * needed are declared here and found in the process.  No allocation. */
#include <stdint.h>
#include <string.h>
#if defined(__x86_64__)
#include <cpuid.h>
#include <immintrin.h>
#endif

#define LGML_API __attribute__((visibility("default")))

typedef struct _object PyObject;
extern PyObject *PyList_GetItem(PyObject *list, intptr_t i);
extern intptr_t PyList_Size(PyObject *list);
extern long long PyLong_AsLongLongAndOverflow(PyObject *v, int *overflow);
extern PyObject *PyErr_Occurred(void);
extern void PyErr_Clear(void);

enum { NOT_INTS = -2 };     /* the caller goes another way */

static int item(PyObject *list, intptr_t i, long long *v) {
    PyObject *o = PyList_GetItem(list, i);
    int over = 0;
    if (o) *v = PyLong_AsLongLongAndOverflow(o, &over);
    if (!o || over || (*v == -1 && PyErr_Occurred())) {
        PyErr_Clear();
        return 0;
    }
    return 1;
}

/* The first n items of a list into dst.  -1, or the place of the first that is not in 0 .. below - 1, or NOT_INTS. */
LGML_API long long lgml_steps_ints(PyObject *list, int32_t *dst, long long n, long long below) {
    if (PyList_Size(list) < n || below > (1LL << 31)) return NOT_INTS;
    for (long long i = 0; i < n; ++i) {
        long long v;
        if (!item(list, i, &v)) return NOT_INTS;
        if (v < 0 || v >= below) return i;
        dst[i] = (int32_t)v;
    }
    return -1;
}

/* positions[N] (first position of its request + place in it), seq_of[N], starts[S + 1], one behind the other */
LGML_API void lgml_steps_rows(int32_t *dst, long long S, const long long *lens, const long long *pos0) {
    long long N = 0;
    for (long long s = 0; s < S; ++s) N += lens[s];
    int32_t *pos = dst, *seq = dst + N, *starts = dst + 2 * N;
    long long at = 0;
    for (long long s = 0; s < S; ++s) {
        starts[s] = (int32_t)at;
        for (long long j = 0; j < lens[s]; ++j, ++at) pos[at] = (int32_t)(pos0[s] + j), seq[at] = (int32_t)s;
    }
    starts[S] = (int32_t)at;
}

/* Rows (request, first token row, tokens, 0) of tiles of at most `tile` tokens of the requests that bring more than `longer_than`; the
 * tile that looks furthest first, ties in the order of the tokens.  The number of tiles. */
LGML_API long long lgml_steps_tiles(int32_t *dst, long long S, const long long *lens, const long long *pos0, long long tile, long long longer_than) {
    long long n = 0, start = 0;
    for (long long s = 0; s < S; start += lens[s++]) {
        if (lens[s] <= longer_than) continue;
        for (long long t = 0; t < lens[s]; t += tile) {
            const long long left = lens[s] - t, tokens = left < tile ? left : tile;
            int32_t *r = dst + 4 * n++;
            r[0] = (int32_t)s, r[1] = (int32_t)(start + t), r[2] = (int32_t)tokens, r[3] = (int32_t)(pos0[s] + t + tokens);
        }
    }
    /* (by insertion: there are a few dozen, and of one request each goes before the last) */
    for (long long i = 1; i < n; ++i) {
        int32_t row[4];
        memcpy(row, dst + 4 * i, sizeof(row));
        long long lo = 0, hi = i;
        while (lo < hi) {
            const long long mid = (lo + hi) / 2;
            if (dst[4 * mid + 3] >= row[3]) lo = mid + 1;
            else hi = mid;
        }
        memmove(dst + 4 * (lo + 1), dst + 4 * lo, (size_t)(i - lo) * sizeof(row));
        memcpy(dst + 4 * lo, row, sizeof(row));
    }
    for (long long i = 0; i < n; ++i) dst[4 * i + 3] = 0;
    return n;
}

/* Rows (first token row, the row past the last) of pieces of at most `piece` tokens of the requests that bring more than `longer_than`, then the
 * first piece of every one of them and the number of pieces, then which requests they are.  Returns the pieces, and the requests in *n_reqs. */
LGML_API long long lgml_steps_pieces(int32_t *dst, long long S, const long long *lens, long long piece, long long longer_than, long long *n_reqs) {
    long long n = 0, R = 0, start = 0;
    for (long long s = 0; s < S; start += lens[s++])
        if (lens[s] > longer_than) {
            ++R;
            for (long long t = 0; t < lens[s]; t += piece, ++n) {
                dst[2 * n] = (int32_t)(start + t);
                dst[2 * n + 1] = (int32_t)(start + (lens[s] - t < piece ? lens[s] : t + piece));
            }
        }
    int32_t *first = dst + 2 * n, *reqs = first + R + 1;
    long long at = 0, r = 0;
    for (long long s = 0; s < S; ++s)
        if (lens[s] > longer_than) {
            first[r] = (int32_t)at, reqs[r++] = (int32_t)s;
            at += (lens[s] + piece - 1) / piece;
        }
    first[r] = (int32_t)at;
    *n_reqs = R;
    return n;
}

/* ---- the keys of pages: SHA-256 (FIPS 180-4) of the key before and the page's tokens as 64-bit little-endian integers ---- */
static const uint32_t K256[64] __attribute__((aligned(16))) = {
    0x428a2f98, 0x71374491, 0xb5c0fbcf, 0xe9b5dba5, 0x3956c25b, 0x59f111f1, 0x923f82a4, 0xab1c5ed5, 0xd807aa98, 0x12835b01, 0x243185be, 0x550c7dc3,
    0x72be5d74, 0x80deb1fe, 0x9bdc06a7, 0xc19bf174, 0xe49b69c1, 0xefbe4786, 0x0fc19dc6, 0x240ca1cc, 0x2de92c6f, 0x4a7484aa, 0x5cb0a9dc, 0x76f988da,
    0x983e5152, 0xa831c66d, 0xb00327c8, 0xbf597fc7, 0xc6e00bf3, 0xd5a79147, 0x06ca6351, 0x14292967, 0x27b70a85, 0x2e1b2138, 0x4d2c6dfc, 0x53380d13,
    0x650a7354, 0x766a0abb, 0x81c2c92e, 0x92722c85, 0xa2bfe8a1, 0xa81a664b, 0xc24b8b70, 0xc76c51a3, 0xd192e819, 0xd6990624, 0xf40e3585, 0x106aa070,
    0x19a4c116, 0x1e376c08, 0x2748774c, 0x34b0bcb5, 0x391c0cb3, 0x4ed8aa4a, 0x5b9cca4f, 0x682e6ff3, 0x748f82ee, 0x78a5636f, 0x84c87814, 0x8cc70208,
    0x90befffa, 0xa4506ceb, 0xbef9a3f7, 0xc67178f2};

static uint32_t ror(uint32_t x, int n) { return x >> n | x << (32 - n); }
static void blocks_plain(uint32_t h[8], const uint8_t *p, size_t n) {
    for (; n--; p += 64) {
        uint32_t w[64], v[8];
        for (int t = 0; t < 16; ++t) w[t] = (uint32_t)p[4 * t] << 24 | (uint32_t)p[4 * t + 1] << 16 | (uint32_t)p[4 * t + 2] << 8 | p[4 * t + 3];
        for (int t = 16; t < 64; ++t) {
            const uint32_t a = w[t - 15], b = w[t - 2];
            w[t] = w[t - 16] + (ror(a, 7) ^ ror(a, 18) ^ a >> 3) + w[t - 7] + (ror(b, 17) ^ ror(b, 19) ^ b >> 10);
        }
        memcpy(v, h, sizeof(v));
        for (int t = 0; t < 64; ++t) {
            const uint32_t t1 = v[7] + (ror(v[4], 6) ^ ror(v[4], 11) ^ ror(v[4], 25)) + ((v[4] & v[5]) ^ (~v[4] & v[6])) + K256[t] + w[t];
            const uint32_t t2 = (ror(v[0], 2) ^ ror(v[0], 13) ^ ror(v[0], 22)) + ((v[0] & v[1]) ^ (v[0] & v[2]) ^ (v[1] & v[2]));
            memmove(v + 1, v, 7 * sizeof(*v));
            v[4] += t1, v[0] = t1 + t2;
        }
        for (int i = 0; i < 8; ++i) h[i] += v[i];
    }
}
#if defined(__x86_64__)
/* The same with the processor's SHA instructions: two rounds an instruction, the state as (A B E F) and (C D G H). */
__attribute__((target("sha,sse4.1,ssse3"))) static void blocks_sha(uint32_t h[8], const uint8_t *p, size_t n) {
    const __m128i turn = _mm_set_epi64x(0x0c0d0e0f08090a0bLL, 0x0405060700010203LL);
    __m128i abef = _mm_set_epi32((int)h[0], (int)h[1], (int)h[4], (int)h[5]), cdgh = _mm_set_epi32((int)h[2], (int)h[3], (int)h[6], (int)h[7]);
    for (; n--; p += 64) {
        const __m128i abef0 = abef, cdgh0 = cdgh;
        __m128i w[4];
        for (int i = 0; i < 4; ++i) w[i] = _mm_shuffle_epi8(_mm_loadu_si128((const __m128i *)(p + 16 * i)), turn);
        /* four rounds with the words x; x then becomes the words 16 on */
#define ROUNDS(t, x)                                                                         \
    do {                                                                                     \
        const __m128i wk = _mm_add_epi32(x, _mm_load_si128((const __m128i *)(K256 + 4 * (t)))); \
        cdgh = _mm_sha256rnds2_epu32(cdgh, abef, wk);                                        \
        abef = _mm_sha256rnds2_epu32(abef, cdgh, _mm_shuffle_epi32(wk, 0x0e));               \
    } while (0)
#define NEXT(x, y, z, u) x = _mm_sha256msg2_epu32(_mm_add_epi32(_mm_sha256msg1_epu32(x, y), _mm_alignr_epi8(u, z, 4)), u)
        for (int t = 0; t < 12; t += 4) {
            ROUNDS(t, w[0]); NEXT(w[0], w[1], w[2], w[3]);
            ROUNDS(t + 1, w[1]); NEXT(w[1], w[2], w[3], w[0]);
            ROUNDS(t + 2, w[2]); NEXT(w[2], w[3], w[0], w[1]);
            ROUNDS(t + 3, w[3]); NEXT(w[3], w[0], w[1], w[2]);
        }
        for (int t = 0; t < 4; ++t) ROUNDS(12 + t, w[t]);
        abef = _mm_add_epi32(abef, abef0), cdgh = _mm_add_epi32(cdgh, cdgh0);
    }
    h[0] = (uint32_t)_mm_extract_epi32(abef, 3), h[1] = (uint32_t)_mm_extract_epi32(abef, 2);
    h[4] = (uint32_t)_mm_extract_epi32(abef, 1), h[5] = (uint32_t)_mm_extract_epi32(abef, 0);
    h[2] = (uint32_t)_mm_extract_epi32(cdgh, 3), h[3] = (uint32_t)_mm_extract_epi32(cdgh, 2);
    h[6] = (uint32_t)_mm_extract_epi32(cdgh, 1), h[7] = (uint32_t)_mm_extract_epi32(cdgh, 0);
}
/* (asked once, when the library is loaded: the instruction that tells takes tens of microseconds in a virtual machine) */
static int has_sha;
__attribute__((constructor)) static void ask(void) {
    unsigned a, b, c, d;
    if (!__get_cpuid_count(7, 0, &a, &b, &c, &d) || !(b >> 29 & 1)) return;
    has_sha = __get_cpuid(1, &a, &b, &c, &d) && (c >> 19 & 1) && (c >> 9 & 1);
}
#else
enum { has_sha = 0 };
#endif

typedef struct {
    uint32_t h[8];
    uint8_t buf[64];
    uint64_t n;
    int plain;
} Hash;

static void blocks(Hash *s, const uint8_t *p, size_t n) {
#if defined(__x86_64__)
    if (!s->plain) {
        blocks_sha(s->h, p, n);
        return;
    }
#endif
    blocks_plain(s->h, p, n);
}
static void start(Hash *s, int plain) {
    static const uint32_t first[8] = {0x6a09e667, 0xbb67ae85, 0x3c6ef372, 0xa54ff53a, 0x510e527f, 0x9b05688c, 0x1f83d9ab, 0x5be0cd19};
    memcpy(s->h, first, sizeof(first));
    s->n = 0, s->plain = plain;
}
static void add(Hash *s, const uint8_t *p, size_t n) {
    size_t have = s->n % 64;
    s->n += n;
    if (have) {
        const size_t part = 64 - have < n ? 64 - have : n;
        memcpy(s->buf + have, p, part);
        p += part, n -= part;
        if (have + part < 64) return;
        blocks(s, s->buf, 1);
    }
    if (n / 64) blocks(s, p, n / 64);
    memcpy(s->buf, p + n / 64 * 64, n % 64);
}
static void finish(Hash *s, uint8_t out[32]) {
    const uint64_t bits = s->n * 8;
    const size_t have = s->n % 64, pad = (have < 56 ? 56 : 120) - have;
    uint8_t tail[72] = {0x80};
    for (int i = 0; i < 8; ++i) tail[pad + i] = (uint8_t)(bits >> (56 - 8 * i));
    add(s, tail, pad + 8);
    for (int i = 0; i < 8; ++i)
        for (int b = 0; b < 4; ++b) out[4 * i + b] = (uint8_t)(s->h[i] >> (24 - 8 * b));
}

/* The keys of pages b0 .. b0 + n - 1 of a token list into out[32 n]; `key` [key_bytes] is the key before them.  0, or NOT_INTS.  `plain`: without the
 * processor's SHA instructions. */
LGML_API int lgml_steps_page_keys(PyObject *list, long long b0, long long n, long long page, const uint8_t *key, long long key_bytes, uint8_t *out, int plain) {
    plain = plain || !has_sha;
    if (PyList_Size(list) < (b0 + n) * page) return NOT_INTS;
    for (long long b = 0; b < n; ++b) {
        Hash s;
        start(&s, plain);
        add(&s, key, (size_t)key_bytes);
        uint8_t raw[64 * 8];
        for (long long at = 0; at < page; at += 64) {
            const long long m = page - at < 64 ? page - at : 64;
            for (long long i = 0; i < m; ++i) {
                long long v;
                if (!item(list, (b0 + b) * page + at + i, &v)) return NOT_INTS;
                for (int k = 0; k < 8; ++k) raw[8 * i + k] = (uint8_t)((uint64_t)v >> (8 * k));
            }
            add(&s, raw, (size_t)(8 * m));
        }
        finish(&s, out + 32 * b);
        key = out + 32 * b, key_bytes = 32;
    }
    return 0;
}

/* ---- launchers called from Python -------------------------------------------------------------------------------------------
 * A callable for a C function of integers, pointers and up to eight floats: ctypes spends 3 us on the arguments of a launch that takes 3 itself.
 * On x86-64 (System V) integers and pointers go in order to six registers and then the stack, floats in order to eight
 * registers of their own, wherever they stand between the integers; what a function does not take it does not look at.  So one call fits all: the
 * integers as 64-bit words in their order, then the floats (of a float the low half of its register counts). */
#if defined(__x86_64__) && defined(__linux__)
typedef struct {
    const char *name;
    PyObject *(*meth)(PyObject *, PyObject *const *, intptr_t);
    int flags;
    const char *doc;
} MethodDef;
extern PyObject *PyCFunction_NewEx(MethodDef *def, PyObject *self, PyObject *module);
extern PyObject *PyLong_FromVoidPtr(void *p);
extern void *PyLong_AsVoidPtr(PyObject *v);
extern long long PyLong_AsLongLong(PyObject *v);
extern PyObject *PyLong_FromLong(long v);
extern double PyFloat_AsDouble(PyObject *v);
extern PyObject *PyTuple_New(intptr_t n);
extern int PyTuple_SetItem(PyObject *t, intptr_t i, PyObject *v);
extern PyObject *PyObject_CallObject(PyObject *f, PyObject *args);
extern void *PyEval_SaveThread(void);
extern void PyEval_RestoreThread(void *state);
extern void Py_IncRef(PyObject *o);
extern void Py_DecRef(PyObject *o);
extern PyObject *PyObject_Type(PyObject *o);
extern char _Py_NoneStruct[];          /* None */
extern char PyLong_Type[];             /* int */
extern void *malloc(size_t n);

enum { MOST_WORDS = 40, MOST_FLOATS = 8, FASTCALL = 0x80 };
typedef long long W;
typedef int (*Launcher)(W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, W, double, double,
                        double, double, double, double, double, double);
typedef struct {
    MethodDef def;
    Launcher fn;
    PyObject *other;        /* takes what is no plain number */
    int n;
    char kinds[MOST_WORDS + MOST_FLOATS + 1];
} Caller;

static int is_int(PyObject *o) {
    PyObject *type = PyObject_Type(o);
    Py_DecRef(type);            /* (lives on: the object holds it) */
    return type == (PyObject *)PyLong_Type;
}

static PyObject *call(PyObject *self, PyObject *const *args, intptr_t n) {
    const Caller *c = (const Caller *)PyLong_AsVoidPtr(self);
    W w[MOST_WORDS] = {0};
    union {
        double d;
        float f;
    } x[MOST_FLOATS] = {{0.0}};
    int nw = 0, nx = 0, ok = n == c->n;
    for (int i = 0; ok && i < n; ++i) {
        if (c->kinds[i] == 'p') {
            /* None, or an int itself: ctypes takes nothing else that could be turned into one */
            if (args[i] == (PyObject *)_Py_NoneStruct) w[nw++] = 0;
            else {
                ok = is_int(args[i]);
                if (ok) w[nw] = PyLong_AsLongLong(args[i]), ok = w[nw++] != -1 || !PyErr_Occurred();
            }
        } else if (c->kinds[i] == 'w') {
            w[nw] = PyLong_AsLongLong(args[i]);
            ok = w[nw++] != -1 || !PyErr_Occurred();
        } else {
            const double v = PyFloat_AsDouble(args[i]);
            ok = v != -1.0 || !PyErr_Occurred();
            if (c->kinds[i] == 'f') x[nx++].f = (float)v;
            else x[nx++].d = v;
        }
    }
    if (!ok) {
        PyErr_Clear();
        PyObject *t = PyTuple_New(n), *got;
        if (!t) return 0;
        for (intptr_t i = 0; i < n; ++i) {
            Py_IncRef(args[i]);
            PyTuple_SetItem(t, i, args[i]);
        }
        got = PyObject_CallObject(c->other, t);
        Py_DecRef(t);
        return got;
    }
    void *state = PyEval_SaveThread();      /* a launch may wait for room in the queue */
    const int rc = c->fn(w[0], w[1], w[2], w[3], w[4], w[5], w[6], w[7], w[8], w[9], w[10], w[11], w[12], w[13], w[14], w[15], w[16], w[17], w[18], w[19],
                         w[20], w[21], w[22], w[23], w[24], w[25], w[26], w[27], w[28], w[29], w[30], w[31], w[32], w[33], w[34], w[35], w[36], w[37], w[38],
                         w[39], x[0].d, x[1].d, x[2].d, x[3].d, x[4].d, x[5].d, x[6].d, x[7].d);
    PyEval_RestoreThread(state);
    return PyLong_FromLong(rc);
}

/* `kinds`: a letter an argument, w (integer), p (pointer), f (float) or d (double).  The function must return an int.  `other` is called instead with
 * arguments that are no numbers, or not as many.  A callable lasts as long as the process; NULL: not here, or too many arguments. */
LGML_API int lgml_steps_caller_fits(const char *kinds) {
    int nw = 0, nx = 0;
    for (const char *k = kinds; *k; ++k) *k == 'w' || *k == 'p' ? ++nw : ++nx;
    return nw <= MOST_WORDS && nx <= MOST_FLOATS;
}
LGML_API PyObject *lgml_steps_caller(void *fn, const char *kinds, PyObject *other) {
    Caller *c = lgml_steps_caller_fits(kinds) ? malloc(sizeof(*c)) : 0;
    if (!c) {
        Py_IncRef((PyObject *)_Py_NoneStruct);
        return (PyObject *)_Py_NoneStruct;
    }
    memset(c, 0, sizeof(*c));
    c->def = (MethodDef){"launcher", call, FASTCALL, 0};
    c->fn = (Launcher)fn, c->other = other, c->n = (int)strlen(kinds);
    memcpy(c->kinds, kinds, (size_t)c->n);
    Py_IncRef(other);
    PyObject *self = PyLong_FromVoidPtr(c);
    PyObject *f = PyCFunction_NewEx(&c->def, self, 0);
    Py_DecRef(self);
    return f;
}
#else
extern char _Py_NoneStruct[];          /* None */
extern void Py_IncRef(PyObject *o);
LGML_API int lgml_steps_caller_fits(const char *kinds) { return kinds == 0; }
LGML_API PyObject *lgml_steps_caller(void *fn, const char *kinds, PyObject *other) {
    (void)fn, (void)kinds, (void)other;
    Py_IncRef((PyObject *)_Py_NoneStruct);
    return (PyObject *)_Py_NoneStruct;
}
#endif
