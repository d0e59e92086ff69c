// The host side of a sampling step, native: what `hydraserve_b200.engine._device` does per row
// and per token around the launch.  A step of a serving loop costs the GPU 10 to 200 us, so a
// microsecond of interpreter per row is the step: packing 256 rows, planning their histogram
// slots and building their results took 550 us in Python (numpy, one dict and one list
// operation per row) next to an 80 us kernel.
//
//   Batch      the packed parameters of one tuple of SamplingParams objects, kept per batch
//              (a serving loop passes the same objects step after step)
//   SlotBook   which request holds which resident histogram slot (a dict for the look-up, an
//              intrusive list for the least-recently-used order)
//   Stepper    one GPU's sampler: plans a step straight into the library's pinned block, runs
//              it without the interpreter lock, turns the records into TokenSample objects
//
// Everything here runs under the interpreter lock except the call into the library.
#define PY_SSIZE_T_CLEAN
#include <Python.h>
#include <structmember.h>

#include <cstddef>
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <unordered_map>
#include <vector>

#include "../../include/hs_sampler.h"

// Whether the interpreter lets small ints be read without a call (Python 3.12 on).  33 histories of up
// to 4,096 tokens: 67,000 reads.
#ifndef HS_COMPACT_INTS
#define HS_COMPACT_INTS (PY_VERSION_HEX >= 0x030C0000)
#endif

namespace {

constexpr uint64_t kSeedStride = 0x1E3779B97F4A7C15ull;  // reference sampling.py:148
constexpr uint64_t kMask63 = 0x7fffffffffffffffull;
// What is kept between calls is bounded, and goes a little at a time: dropping a batch can mean freeing
// its parameter objects, 60 ns each, in whichever call comes next.
constexpr size_t kBatchesMax = 64;
constexpr size_t kBatchRowsMax = 4096;  // over all kept batches
constexpr size_t kRowsMax = 8192;

// Python objects this module works with, handed over once by bind().
struct Bound {
  PyObject* token_sample = nullptr;    // the TokenSample type
  Py_ssize_t off_token = 0, off_logprob = 0, off_top = 0;  // its slots
  PyObject* as_int64 = nullptr;        // any sequence of numbers -> contiguous 1-D int64 buffer
  PyObject* unseeded_keys = nullptr;   // params -> stream key or None per row
  PyObject* neg_inf = nullptr;
  PyObject* empty = nullptr;
} g;

// Attribute names, interned.
PyObject *s_temperature, *s_top_p, *s_top_k, *s_min_p, *s_repetition, *s_presence, *s_frequency, *s_seed, *s_logprobs;

struct Ref {  // an owned reference
  PyObject* p;
  explicit Ref(PyObject* o = nullptr) : p(o) {}
  ~Ref() { Py_XDECREF(p); }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  Ref(Ref&& o) noexcept : p(o.p) { o.p = nullptr; }
  PyObject* take() { PyObject* o = p; p = nullptr; return o; }
  explicit operator bool() const { return p != nullptr; }
};

// ---- parameters ------------------------------------------------------------------------------
struct Row {  // what one SamplingParams object comes to
  hs_row_params p;
  int logprobs;     // as asked for, -1 = none
  bool penalised, greedy, seeded, zero_t;
  uint64_t seed;
};

bool number(PyObject* o, PyObject* name, double& out) {
  Ref v(PyObject_GetAttr(o, name));
  if (!v) return false;
  out = PyFloat_AsDouble(v.p);
  return !(out == -1.0 && PyErr_Occurred());
}

bool pack_row(PyObject* o, Row& r) {
  std::memset(&r, 0, sizeof r);
  double t, top_p, min_p, rep, pres, freq;
  if (!number(o, s_temperature, t) || !number(o, s_top_p, top_p) || !number(o, s_min_p, min_p) ||
      !number(o, s_repetition, rep) || !number(o, s_presence, pres) || !number(o, s_frequency, freq))
    return false;
  Ref k(PyObject_GetAttr(o, s_top_k)), seed(PyObject_GetAttr(o, s_seed)), lp(PyObject_GetAttr(o, s_logprobs));
  if (!k || !seed || !lp) return false;
  Ref k_int(PyNumber_Long(k.p));
  if (!k_int) return false;
  int over = 0;
  const long long kk = PyLong_AsLongLongAndOverflow(k_int.p, &over);
  if (kk == -1 && !over && PyErr_Occurred()) return false;
  r.p.temperature = (float)t; r.p.top_p = (float)top_p; r.p.min_p = (float)min_p;
  r.p.repetition_penalty = (float)rep; r.p.presence_penalty = (float)pres; r.p.frequency_penalty = (float)freq;
  r.p.top_k = over > 0 || kk > 0x7fffffffll ? 0x7fffffff : (int32_t)kk;
  r.logprobs = -1;
  if (lp.p != Py_None) {
    const long v = PyLong_AsLong(lp.p);
    if (v == -1 && PyErr_Occurred()) return false;
    r.logprobs = (int)v;
  }
  r.p.n_logprobs = r.logprobs;
  r.penalised = !(rep == 1.0 && pres == 0.0 && freq == 0.0);           // reference sampling.py:94-99
  r.greedy = t == 0.0 && r.logprobs < 0 && !r.penalised;               // reference sampling.py:86-91
  r.p.flags = r.greedy ? HS_ROW_PLAIN_GREEDY : 0u;
  r.p.slot = -1;
  r.zero_t = t == 0.0;
  r.seeded = seed.p != Py_None || r.zero_t;
  if (seed.p != Py_None) {
    Ref i(PyNumber_Index(seed.p));
    if (!i) return false;
    r.seed = PyLong_AsUnsignedLongLongMask(i.p);
    if (r.seed == (uint64_t)-1 && PyErr_Occurred()) return false;
  }
  return true;
}

struct RowEntry { PyObject* owner; Row row; };
// By object; the reference keeps the address its own.  (Both caches live as long as the process:
// nothing of theirs may be released once the interpreter is gone.)
auto& g_rows = *new std::unordered_map<PyObject*, RowEntry>();
auto& g_rows_order = *new std::vector<PyObject*>();
size_t g_rows_next = 0;

const Row* row_of(PyObject* o) {
  auto it = g_rows.find(o);
  if (it != g_rows.end()) return &it->second.row;
  Row r;
  if (!pack_row(o, r)) return nullptr;
  Py_INCREF(o);
  PyObject* gone = nullptr;  // the one that has been here longest
  if (g_rows_order.size() < kRowsMax) {
    g_rows_order.push_back(o);
  } else {
    gone = g_rows_order[g_rows_next];
    g_rows_order[g_rows_next] = o;
    g_rows_next = (g_rows_next + 1) % kRowsMax;
    g_rows.erase(gone);
  }
  const Row* kept = &(g_rows[o] = RowEntry{o, r}).row;
  Py_XDECREF(gone);  // (last: this may run any code)
  return kept;
}

// A batch's parameters.  `view` is what Python sees: (the params, packed static part, any
// unseeded row, seeds or None, which rows have penalties).
struct Batch {
  PyObject* view = nullptr;
  std::vector<PyObject*> key;       // the params objects (kept alive by view)
  std::vector<hs_row_params> rows;  // static part: seed and slot are filled in per call
  std::vector<uint64_t> seeds;
  std::vector<int8_t> logprobs;
  std::vector<uint8_t> penalised;
  bool all_greedy = true, any_unseeded = false, any_penalised = false, any_logprobs = false, any_zero_t = false;
  int top_k_lo = 0x7fffffff, top_k_hi = 0;  // over all rows
  uint64_t used = 0;
  Batch() = default;
  Batch(const Batch&) = delete;
  Batch& operator=(const Batch&) = delete;
  ~Batch() { Py_XDECREF(view); }
};
// (shared: a call keeps its batch when another one pushes it out of the cache meanwhile)
typedef std::shared_ptr<Batch> BatchRef;
auto& g_batches = *new std::unordered_multimap<uint64_t, BatchRef>();
uint64_t g_batch_clock = 0;
size_t g_batch_rows = 0;  // of the kept batches

PyObject* batch_view(const Batch& b) {
  const Py_ssize_t n = (Py_ssize_t)b.key.size();
  Ref params(PyTuple_New(n)), pen(PyTuple_New(n));
  if (!params || !pen) return nullptr;
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyTuple_SET_ITEM(params.p, i, Py_NewRef(b.key[(size_t)i]));
    PyTuple_SET_ITEM(pen.p, i, Py_NewRef(b.penalised[(size_t)i] ? Py_True : Py_False));
  }
  Ref rows(PyBytes_FromStringAndSize(reinterpret_cast<const char*>(b.rows.data()), n * (Py_ssize_t)sizeof(hs_row_params)));
  Ref seeds(b.any_unseeded ? Py_NewRef(Py_None)
                           : PyBytes_FromStringAndSize(reinterpret_cast<const char*>(b.seeds.data()), n * 8));
  if (!rows || !seeds) return nullptr;
  return PyTuple_Pack(5, params.p, rows.p, b.any_unseeded ? Py_True : Py_False, seeds.p, pen.p);
}

// The batch of a list or tuple of SamplingParams (items / n as PySequence_Fast gives them).
BatchRef batch_of(PyObject** items, Py_ssize_t n) {
  uint64_t h = 0x9E3779B97F4A7C15ull ^ (uint64_t)n;
  for (Py_ssize_t i = 0; i < n; ++i) h = (h ^ ((uint64_t)(uintptr_t)items[i] >> 4)) * 0x100000001B3ull;
  auto range = g_batches.equal_range(h);
  for (auto it = range.first; it != range.second; ++it) {
    const BatchRef& b = it->second;
    if ((Py_ssize_t)b->key.size() == n && (n == 0 || std::memcmp(b->key.data(), items, (size_t)n * sizeof(PyObject*)) == 0)) {
      b->used = ++g_batch_clock;
      return b;
    }
  }
  BatchRef b = std::make_shared<Batch>();
  // (attributes are read under the lock, and a property could run anything: work on a copy)
  b->key.assign(items, items + n);
  for (PyObject* o : b->key) Py_INCREF(o);
  bool ok = true;
  for (Py_ssize_t i = 0; ok && i < n; ++i) {
    const Row* r = row_of(b->key[(size_t)i]);
    if (!r) { ok = false; break; }
    b->rows.push_back(r->p);
    b->seeds.push_back(r->seed);
    b->logprobs.push_back((int8_t)r->logprobs);
    b->penalised.push_back(r->penalised ? 1 : 0);
    b->all_greedy = b->all_greedy && r->greedy;
    b->any_unseeded = b->any_unseeded || !r->seeded;
    b->any_penalised = b->any_penalised || r->penalised;
    b->any_logprobs = b->any_logprobs || r->logprobs >= 0;
    b->any_zero_t = b->any_zero_t || r->zero_t;
    b->top_k_lo = std::min(b->top_k_lo, r->p.top_k);
    b->top_k_hi = std::max(b->top_k_hi, r->p.top_k);
  }
  if (ok) b->view = batch_view(*b);
  for (PyObject* o : b->key) Py_DECREF(o);  // (view holds them now)
  if (!ok || !b->view) return nullptr;
  std::vector<BatchRef> gone;  // the least recently used ones (let go of at the end: this may run any code)
  while (!g_batches.empty() && (g_batches.size() >= kBatchesMax || g_batch_rows + (size_t)n > kBatchRowsMax)) {
    auto oldest = g_batches.begin();
    for (auto it = g_batches.begin(); it != g_batches.end(); ++it)
      if (it->second->used < oldest->second->used) oldest = it;
    g_batch_rows -= oldest->second->key.size();
    gone.push_back(oldest->second);
    g_batches.erase(oldest);
  }
  b->used = ++g_batch_clock;
  g_batch_rows += (size_t)n;
  g_batches.emplace(h, b);
  return b;
}

// step -> the seed the kernels take: (seed + (step + 1) * stride) mod 2^63
bool mix_seeds(const Batch& b, PyObject** steps, PyObject* keys, hs_row_params* out) {
  const size_t n = b.rows.size();
  for (size_t i = 0; i < n; ++i) {
    long long step;
    if (PyLong_Check(steps[i])) {
      step = PyLong_AsLongLong(steps[i]);
    } else {
      Ref v(PyNumber_Long(steps[i]));
      if (!v) return false;
      step = PyLong_AsLongLong(v.p);
    }
    if (step == -1 && PyErr_Occurred()) return false;
    uint64_t seed = b.seeds[i];
    if (keys && keys != Py_None) {
      // a row without a seed of its own takes the key it is given
      Ref k(PySequence_GetItem(keys, (Py_ssize_t)i));
      if (!k) return false;
      if (k.p != Py_None) {
        PyObject* own = PyTuple_GET_ITEM(PyTuple_GET_ITEM(b.view, 0), (Py_ssize_t)i);
        Ref has(PyObject_GetAttr(own, s_seed));
        if (!has) return false;
        if (has.p == Py_None) {
          seed = PyLong_AsUnsignedLongLongMask(k.p);
          if (seed == (uint64_t)-1 && PyErr_Occurred()) return false;
        }
      }
    }
    out[i].seed = (seed + ((uint64_t)step + 1ull) * kSeedStride) & kMask63;
  }
  return true;
}

// ---- requests and their slots ------------------------------------------------------------------
struct SlotEntry {
  PyObject_HEAD
  PyObject* request;     // owned while the entry is in a book
  SlotEntry *prev, *next;  // LRU list of the book, oldest first
  uint64_t call;         // the last call that planned it
  uint64_t appended;     // the last call that appended to it
  int slot;              // -1 once evicted or released
  long long counted;     // tokens of the history the device has counted
};

PyObject* entry_item(PyObject* self, Py_ssize_t i) {
  auto* e = reinterpret_cast<SlotEntry*>(self);
  if (i == 0) return PyLong_FromLong(e->slot);
  if (i == 1) return PyLong_FromLongLong(e->counted);
  PyErr_SetString(PyExc_IndexError, "an entry is (slot, tokens counted)");
  return nullptr;
}
int entry_set(PyObject* self, Py_ssize_t i, PyObject* v) {
  auto* e = reinterpret_cast<SlotEntry*>(self);
  if (i != 1 || !v) {
    PyErr_SetString(PyExc_IndexError, "only the tokens counted can be set");
    return -1;
  }
  const long long n = PyLong_AsLongLong(v);
  if (n == -1 && PyErr_Occurred()) return -1;
  e->counted = n;
  return 0;
}
Py_ssize_t entry_len(PyObject*) { return 2; }
// (a request id can be any object, so entries and books take part in cycle collection)
int entry_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<SlotEntry*>(self)->request);
  return 0;
}
void entry_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  Py_XDECREF(reinterpret_cast<SlotEntry*>(self)->request);
  PyObject_GC_Del(self);
}
PySequenceMethods entry_seq{};
PyTypeObject SlotEntryType = {PyVarObject_HEAD_INIT(nullptr, 0)};

struct SlotBook {
  PyObject_HEAD
  int n_slots;
  PyObject* entries;         // request id -> SlotEntry
  std::vector<int>* free_;
  SlotEntry *oldest, *newest;
  uint64_t calls;            // calls planned on this book
};
PyTypeObject SlotBookType = {PyVarObject_HEAD_INIT(nullptr, 0)};

void unlink(SlotBook* b, SlotEntry* e) {
  (e->prev ? e->prev->next : b->oldest) = e->next;
  (e->next ? e->next->prev : b->newest) = e->prev;
  e->prev = e->next = nullptr;
}
void link_newest(SlotBook* b, SlotEntry* e) {
  e->prev = b->newest;
  e->next = nullptr;
  (b->newest ? b->newest->next : b->oldest) = e;
  b->newest = e;
}
void touch(SlotBook* b, SlotEntry* e) {
  if (b->newest == e) return;
  unlink(b, e);
  link_newest(b, e);
}
// The entry leaves the book; its slot is free again.
bool drop(SlotBook* b, SlotEntry* e) {
  Ref hold(Py_NewRef(reinterpret_cast<PyObject*>(e)));
  if (PyDict_DelItem(b->entries, e->request) < 0) return false;
  unlink(b, e);
  b->free_->push_back(e->slot);
  e->slot = -1;
  e->counted = 0;
  return true;
}
SlotEntry* find(SlotBook* b, PyObject* request) {  // borrowed; nullptr without an error = not there
  return reinterpret_cast<SlotEntry*>(PyDict_GetItemWithError(b->entries, request));
}
SlotEntry* add(SlotBook* b, PyObject* request) {  // borrowed; a free slot is there
  SlotEntry* e = PyObject_GC_New(SlotEntry, &SlotEntryType);
  if (!e) return nullptr;
  e->request = Py_NewRef(request);
  e->prev = e->next = nullptr;
  e->call = e->appended = 0;
  e->slot = b->free_->back();
  e->counted = 0;
  PyObject_GC_Track(reinterpret_cast<PyObject*>(e));
  const int rc = PyDict_SetItem(b->entries, request, reinterpret_cast<PyObject*>(e));
  Py_DECREF(e);  // (the book's dict holds it)
  if (rc < 0) return nullptr;
  b->free_->pop_back();
  link_newest(b, e);
  return e;
}

PyObject* book_new(PyTypeObject* type, PyObject*, PyObject*) {
  auto* b = reinterpret_cast<SlotBook*>(type->tp_alloc(type, 0));
  if (!b) return nullptr;
  b->entries = PyDict_New();
  b->free_ = new std::vector<int>();
  if (!b->entries) { Py_DECREF(b); return nullptr; }
  return reinterpret_cast<PyObject*>(b);
}
int book_init(PyObject* self, PyObject* args, PyObject*) {
  auto* b = reinterpret_cast<SlotBook*>(self);
  int n = 0;
  if (!PyArg_ParseTuple(args, "i", &n)) return -1;
  b->n_slots = n;
  b->free_->clear();
  for (int s = n - 1; s >= 0; --s) b->free_->push_back(s);
  return 0;
}
int book_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<SlotBook*>(self)->entries);
  return 0;
}
int book_clear(PyObject* self) {
  // (the list runs through entries the dict is about to let go of)
  auto* b = reinterpret_cast<SlotBook*>(self);
  b->oldest = b->newest = nullptr;
  if (b->entries) PyDict_Clear(b->entries);
  return 0;
}
void book_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  auto* b = reinterpret_cast<SlotBook*>(self);
  Py_XDECREF(b->entries);
  delete b->free_;
  Py_TYPE(self)->tp_free(self);
}
PyObject* book_release(PyObject* self, PyObject* request) {
  auto* b = reinterpret_cast<SlotBook*>(self);
  SlotEntry* e = find(b, request);
  if (!e) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_FALSE;
  }
  if (!drop(b, e)) return nullptr;
  Py_RETURN_TRUE;
}
PyMethodDef book_methods[] = {
    {"release", book_release, METH_O, "Forget a request; True if it held a slot."},
    {nullptr, nullptr, 0, nullptr}};
PyMemberDef book_members[] = {
    {"n_slots", T_INT, offsetof(SlotBook, n_slots), READONLY, "resident slots"},
    {"entries", T_OBJECT_EX, offsetof(SlotBook, entries), READONLY, "request id -> (slot, tokens counted)"},
    {nullptr, 0, 0, 0, nullptr}};

// ---- planning a step -------------------------------------------------------------------------------
struct Append {
  int slot;
  PyObject* history;       // borrowed from the call's histories
  long long from, count;   // tokens history[from : from + count]
};
struct StepPlan {
  std::vector<int> resets;
  std::vector<Append> appends;
  std::vector<Ref> entries;  // the book's entries among them
  bool repeats = false;      // a slot is appended to twice
};

inline Py_ssize_t length(PyObject* h) {
  if (PyList_CheckExact(h)) return PyList_GET_SIZE(h);
  if (PyTuple_CheckExact(h)) return PyTuple_GET_SIZE(h);
  return PyObject_Length(h);
}

// Slot per row (slots[i], -1 = none), and the resets and appends that bring the device up to
// date.  A penalised row whose history is empty goes without a slot, with and without a
// request id, so that the same kernel path serves it either way; the request keeps the slot
// it was given.
bool plan_step(SlotBook* book, int per_call_base, const Batch& b, PyObject** histories, PyObject* ids, int* slots,
               StepPlan& plan) {
  const Py_ssize_t n = (Py_ssize_t)b.key.size();
  const uint64_t call = ++book->calls;
  bool marked = false;
  for (Py_ssize_t i = 0; i < n; ++i) {
    slots[i] = -1;
    if (!b.penalised[(size_t)i]) continue;
    const long long len = length(histories[i]);
    if (len < 0) return false;
    PyObject* id = ids ? PySequence_Fast_GET_ITEM(ids, i) : Py_None;
    SlotEntry* e = nullptr;
    if (id != Py_None) {
      e = find(book, id);
      if (!e && PyErr_Occurred()) return false;
      bool is_new = false;
      if (!e) {
        if (book->free_->empty()) {
          // never a request of this call: mark those that hold a slot, then take the oldest other
          if (!marked) {
            for (Py_ssize_t j = 0; j < n; ++j) {
              PyObject* other = PySequence_Fast_GET_ITEM(ids, j);
              if (other == Py_None) continue;
              SlotEntry* o = find(book, other);
              if (!o && PyErr_Occurred()) return false;
              if (o) o->call = call;
            }
            marked = true;
          }
          SlotEntry* v = book->oldest;
          while (v && v->call == call) v = v->next;
          if (v && !drop(book, v)) return false;
        }
        if (!book->free_->empty()) {
          e = add(book, id);
          if (!e) return false;
          is_new = true;
        }
      } else {
        touch(book, e);
      }
      if (e) {
        e->call = call;
        if (is_new || len != e->counted) plan.entries.emplace_back(Py_NewRef(reinterpret_cast<PyObject*>(e)));
        if (is_new || len < e->counted) {  // (a history that got shorter is counted anew)
          plan.resets.push_back(e->slot);
          e->counted = 0;
        }
        if (len > e->counted) {
          if (e->appended == call) plan.repeats = true;
          e->appended = call;
          plan.appends.push_back(Append{e->slot, histories[i], e->counted, len - e->counted});
          e->counted = len;
        }
        if (len > 0) slots[i] = e->slot;
        continue;
      }
    }
    if (len == 0) continue;
    const int slot = per_call_base + (int)i;
    plan.resets.push_back(slot);
    plan.appends.push_back(Append{slot, histories[i], 0, len});
    slots[i] = slot;
  }
  return true;
}

// history[from : from + count] of anything that has a length
PyObject* tail_of(const Append& a) {
  if (a.from == 0) return Py_NewRef(a.history);  // (planned with its whole length)
  Ref seq(PySequence_Check(a.history) || PyMapping_Check(a.history) ? Py_NewRef(a.history) : PySequence_Tuple(a.history));
  Ref lo(PyLong_FromLongLong(a.from)), hi(PyLong_FromLongLong(a.from + a.count));
  if (!seq || !lo || !hi) return nullptr;
  Ref range(PySlice_New(lo.p, hi.p, nullptr));
  return range ? PyObject_GetItem(seq.p, range.p) : nullptr;
}

inline int32_t device_token(long long t, int vocab) {
  // the kernels ignore ids outside the vocabulary (reference sampling.py:108); -1 stands for them
  return t < 0 || t >= vocab ? -1 : (int32_t)t;
}

// Tokens of one append into out[0 .. count).  Lists and tuples of ints are read in place.
bool gather(const Append& a, int vocab, int32_t* out) {
  PyObject* h = a.history;
  const bool list = PyList_CheckExact(h);
  if (length(h) < a.from + a.count) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_RuntimeError, "a history got shorter while its step was being prepared");
    return false;
  }
  if (list || PyTuple_CheckExact(h)) {
    PyObject* const* items = (list ? reinterpret_cast<PyListObject*>(h)->ob_item
                                   : reinterpret_cast<PyTupleObject*>(h)->ob_item) + a.from;
    long long i = 0;
    for (; i < a.count; ++i) {
      // (a long history's int objects lie all over the heap: ask for them ahead)
      if (i + 16 < a.count) __builtin_prefetch(items[i + 16]);
      PyObject* o = items[i];
      if (!PyLong_CheckExact(o)) break;
#if HS_COMPACT_INTS
      const PyLongObject* l = reinterpret_cast<const PyLongObject*>(o);
      if (PyUnstable_Long_IsCompact(l)) {
        out[i] = device_token((long long)PyUnstable_Long_CompactValue(l), vocab);
      } else
#endif
      {
        int over = 0;
        const long long t = PyLong_AsLongLongAndOverflow(o, &over);
        if (over) {
          PyErr_SetString(PyExc_OverflowError, "token id too large to convert to 64 bits");
          return false;
        }
        out[i] = device_token(t, vocab);
      }
    }
    if (i == a.count) return true;
  }
  // anything else (arrays, other number types): through numpy
  Ref tail(tail_of(a));
  if (!tail) return false;
  Ref flat(PyObject_CallOneArg(g.as_int64, tail.p));
  if (!flat) return false;
  Py_buffer view;
  if (PyObject_GetBuffer(flat.p, &view, PyBUF_C_CONTIGUOUS) < 0) return false;
  const bool fits = view.itemsize == 8 && view.len == a.count * 8;
  if (fits)
    for (long long i = 0; i < a.count; ++i) out[i] = device_token(static_cast<const int64_t*>(view.buf)[i], vocab);
  PyBuffer_Release(&view);
  if (!fits) PyErr_SetString(PyExc_ValueError, "a history must be a flat sequence of token ids");
  return fits;
}

// ---- results -----------------------------------------------------------------------------------------
inline PyObject** slot_at(PyObject* o, Py_ssize_t offset) {
  return reinterpret_cast<PyObject**>(reinterpret_cast<char*>(o) + offset);
}
// TokenSample objects without the frozen dataclass's __init__.
// A step's results are made in two parts: the objects while the GPU is at work, then, from the
// records, the numbers in them (1,024 samples: 30 of 42 us pass before the records are there).
// They hold numbers and tuples of numbers only, so they cannot be part of a cycle: the collector need
// not look at the thousands of them a step makes.
PyObject* blank_pairs(int n) {  // ((id, value), ...), to be filled in
  if (n == 0) return Py_NewRef(g.empty);
  Ref top(PyTuple_New(n));
  for (int i = 0; top && i < n; ++i) {
    PyObject* t = PyTuple_New(2);
    if (!t) return nullptr;
    PyObject_GC_UnTrack(t);
    PyTuple_SET_ITEM(top.p, i, t);
  }
  if (top) PyObject_GC_UnTrack(top.p);
  return top.take();
}
bool blank_sample(PyObject* out, Py_ssize_t i, int asked, int vocab) {
  auto* type = reinterpret_cast<PyTypeObject*>(g.token_sample);
  PyObject* o = type->tp_alloc(type, 0);
  if (!o) return false;
  if (PyObject_GC_IsTracked(o)) PyObject_GC_UnTrack(o);
  PyTuple_SET_ITEM(out, i, o);
  if (asked < 0) *slot_at(o, g.off_logprob) = Py_NewRef(Py_None);
  PyObject* top = blank_pairs(asked < 0 ? 0 : std::min(asked, vocab));
  if (!top) return false;
  *slot_at(o, g.off_top) = top;
  return true;
}
PyObject* blank_samples(Py_ssize_t n, const int8_t* logprobs, int vocab) {
  Ref out(PyTuple_New(n));
  if (!out) return nullptr;
  for (Py_ssize_t i = 0; i < n; ++i)
    if (!blank_sample(out.p, i, logprobs ? logprobs[i] : -1, vocab)) return nullptr;
  if (n) PyObject_GC_UnTrack(out.p);
  return out.take();
}
inline bool set_token(PyObject* sample, int32_t token) {
  return (*slot_at(sample, g.off_token) = PyLong_FromLong(token)) != nullptr;
}
bool fill_sample(PyObject* o, const hs_row_out& r, int asked, int vocab) {
  if (!set_token(o, r.token)) return false;
  if (asked < 0) return true;
  if (!(*slot_at(o, g.off_logprob) = PyFloat_FromDouble((double)r.logprob))) return false;
  PyObject* top = *slot_at(o, g.off_top);
  const int want = std::min(asked, vocab);
  const int n = std::max(0, std::min((int)r.n_top, want));
  auto set = [&](int at, int id, PyObject* value) {
    PyObject* t = PyTuple_GET_ITEM(top, at);
    PyObject* i = PyLong_FromLong(id);
    PyTuple_SET_ITEM(t, 0, i);
    PyTuple_SET_ITEM(t, 1, value);
    return i && value;
  };
  int at = 0;
  for (; at < n; ++at)
    if (!set(at, r.top_ids[at], PyFloat_FromDouble((double)r.top_logprobs[at]))) return false;
  // fewer candidates than requested: the reference lists filtered ids at -inf
  for (int id = 0; at < want; ++id) {
    bool taken = false;
    for (int j = 0; j < n; ++j) taken = taken || r.top_ids[j] == id;
    if (!taken && !set(at++, id, Py_NewRef(g.neg_inf))) return false;
  }
  return true;
}
PyObject* filled_samples(Ref& out, const hs_row_out* rec, const Batch& b, int vocab) {
  for (Py_ssize_t i = 0; i < (Py_ssize_t)b.key.size(); ++i)
    if (!fill_sample(PyTuple_GET_ITEM(out.p, i), rec[i], b.logprobs[(size_t)i], vocab)) return nullptr;
  return out.take();
}
PyObject* samples_of(const hs_row_out* rec, const Batch& b, int vocab) {
  Ref out(blank_samples((Py_ssize_t)b.key.size(), b.logprobs.data(), vocab));
  return out ? filled_samples(out, rec, b, vocab) : nullptr;
}

// ---- the stepper ---------------------------------------------------------------------------------------
typedef int (*BlockFn)(hs_sampler*, size_t, void**);
typedef int (*StepFn)(hs_sampler*, const void*, int, int64_t, int, int, const hs_step_desc*, const hs_row_out**, void*);
typedef int (*GreedyFn)(hs_sampler*, const void*, int, int64_t, int, int, const int32_t**, void*);
typedef int (*WaitFn)(hs_sampler*, void*);
typedef const char* (*TextFn)(hs_sampler*);

struct Stepper {
  PyObject_HEAD
  hs_sampler* h;    // null once closed
  PyObject* book;
  PyObject* error;  // the exception type
  int per_call_base;
  BlockFn block;
  StepFn step;
  GreedyFn greedy;
  WaitFn wait;
  TextFn text;
};
PyTypeObject StepperType = {PyVarObject_HEAD_INIT(nullptr, 0)};

PyObject* stepper_new(PyTypeObject* type, PyObject* args, PyObject*) {
  unsigned long long h, block, step, greedy, wait, text;
  PyObject *book, *error;
  int base;
  if (!PyArg_ParseTuple(args, "KO!iOKKKKK", &h, &SlotBookType, &book, &base, &error, &block, &step, &greedy, &wait, &text)) return nullptr;
  auto* s = reinterpret_cast<Stepper*>(type->tp_alloc(type, 0));
  if (!s) return nullptr;
  s->h = reinterpret_cast<hs_sampler*>(h);
  s->book = Py_NewRef(book);
  s->error = Py_NewRef(error);
  s->per_call_base = base;
  s->block = reinterpret_cast<BlockFn>(block);
  s->step = reinterpret_cast<StepFn>(step);
  s->greedy = reinterpret_cast<GreedyFn>(greedy);
  s->wait = reinterpret_cast<WaitFn>(wait);
  s->text = reinterpret_cast<TextFn>(text);
  return reinterpret_cast<PyObject*>(s);
}
int stepper_traverse(PyObject* self, visitproc visit, void* arg) {
  Py_VISIT(reinterpret_cast<Stepper*>(self)->book);
  Py_VISIT(reinterpret_cast<Stepper*>(self)->error);
  return 0;
}
void stepper_dealloc(PyObject* self) {
  PyObject_GC_UnTrack(self);
  auto* s = reinterpret_cast<Stepper*>(self);
  Py_XDECREF(s->book);
  Py_XDECREF(s->error);
  Py_TYPE(self)->tp_free(self);
}
PyObject* failed(Stepper* s, const char* what, int status) {
  PyErr_Format(s->error, "%s: (%d) %s", what, status, s->text(s->h));
  return nullptr;
}

// close(): the sampler is about to be destroyed; later steps fail.
PyObject* stepper_close(PyObject* self, PyObject*) {
  reinterpret_cast<Stepper*>(self)->h = nullptr;
  Py_RETURN_NONE;
}

inline size_t up16(size_t v) { return (v + 15) & ~size_t(15); }

// What a failed step leaves behind: the histograms it was to empty or bring up to date may not be, so
// their requests start over.
void forget(SlotBook* book, const StepPlan& plan) {
  PyObject *type, *value, *trace;
  PyErr_Fetch(&type, &value, &trace);
  for (const Ref& r : plan.entries) {
    auto* e = reinterpret_cast<SlotEntry*>(r.p);
    if (e->slot >= 0 && !drop(book, e)) PyErr_Clear();
  }
  PyErr_Restore(type, value, trace);
}

// step(logits address, dtype, row stride, vocabulary, histories, params, steps, request ids or
// None, stream, packed) -> tuple of TokenSample, or (packed) (records, log-probabilities asked for).
// When a row needs more than this call can give (a status, rows for the general kernel) the
// answer is a list instead: [records, params], as bytearrays, for the caller to sort out.
PyObject* stepper_step(PyObject* self, PyObject* const* args, Py_ssize_t n_args) {
  auto* s = reinterpret_cast<Stepper*>(self);
  if (n_args != 10) {
    PyErr_SetString(PyExc_TypeError, "step takes ten arguments");
    return nullptr;
  }
  if (!s->h) return failed(s, "hs_step", HS_ERR_INVALID);
  const void* logits = reinterpret_cast<const void*>((uintptr_t)PyLong_AsUnsignedLongLong(args[0]));
  const int dtype = (int)PyLong_AsLong(args[1]);
  const int64_t stride = PyLong_AsLongLong(args[2]);
  const int vocab = (int)PyLong_AsLong(args[3]);
  void* stream = reinterpret_cast<void*>((uintptr_t)PyLong_AsUnsignedLongLong(args[8]));
  const int packed = PyObject_IsTrue(args[9]);
  if (PyErr_Occurred()) return nullptr;
  // (own copies: what the caller passed may be changed by code that runs meanwhile)
  Ref histories(PySequence_Tuple(args[4])), params(PySequence_Tuple(args[5])), steps(PySequence_Tuple(args[6]));
  if (!histories || !params || !steps) return nullptr;
  Ref ids(args[7] == Py_None ? nullptr : PySequence_Tuple(args[7]));
  if (!ids && args[7] != Py_None) return nullptr;
  const Py_ssize_t n = PyTuple_GET_SIZE(params.p);
  if (PyTuple_GET_SIZE(histories.p) != n || PyTuple_GET_SIZE(steps.p) != n || (ids && PyTuple_GET_SIZE(ids.p) != n)) {
    PyErr_SetString(PyExc_ValueError, "sampling metadata must match the logits batch");
    return nullptr;
  }
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(params.p)->ob_item, n);
  if (!b) return nullptr;
  Ref keys(b->any_unseeded ? PyObject_CallOneArg(g.unseeded_keys, params.p) : nullptr);
  if (!keys && b->any_unseeded) return nullptr;

  StepPlan plan;
  std::vector<int> slots((size_t)n, -1);
  auto* book = reinterpret_cast<SlotBook*>(s->book);
  if (b->any_penalised) {
    if (!plan_step(book, s->per_call_base, *b, reinterpret_cast<PyTupleObject*>(histories.p)->ob_item,
                   ids ? ids.p : nullptr, slots.data(), plan)) {
      forget(book, plan);
      return nullptr;
    }
  }
  // the block: parameters, then (if anything is to be counted) resets, slots, offsets, tokens
  hs_step_desc d;
  std::memset(&d, 0, sizeof d);
  long long total = 0, longest = 0;
  for (const Append& a : plan.appends) {
    total += a.count;
    if (a.count > longest) longest = a.count;
  }
  if (total > 0x7fffffffll) {
    forget(book, plan);
    PyErr_SetString(PyExc_ValueError, "too many history tokens in one step");
    return nullptr;
  }
  size_t at = up16((size_t)n * sizeof(hs_row_params));
  d.n_resets = (int32_t)plan.resets.size();
  d.n_appends = (int32_t)plan.appends.size();
  d.max_tokens = (int32_t)longest;
  d.repeats = plan.repeats ? 1 : 0;
  d.resets_at = at; at += up16(plan.resets.size() * 4);
  d.slots_at = at; at += up16(plan.appends.size() * 4);
  d.offsets_at = at; at += up16((plan.appends.size() + 1) * 4);
  d.tokens_at = at; at += up16((size_t)total * 4);
  d.bytes = at;
  void* block = nullptr;
  int st = s->block(s->h, at, &block);
  if (st != HS_OK) {
    forget(book, plan);
    return failed(s, "hs_step_block", st);
  }
  auto* base = static_cast<unsigned char*>(block);
  auto* rows = reinterpret_cast<hs_row_params*>(base);
  std::memcpy(rows, b->rows.data(), (size_t)n * sizeof(hs_row_params));
  bool ok = mix_seeds(*b, reinterpret_cast<PyTupleObject*>(steps.p)->ob_item, keys.p, rows);
  for (Py_ssize_t i = 0; i < n; ++i) rows[i].slot = slots[(size_t)i];
  if (!plan.resets.empty()) std::memcpy(base + d.resets_at, plan.resets.data(), plan.resets.size() * 4);
  {
    auto* slot_list = reinterpret_cast<int32_t*>(base + d.slots_at);
    auto* offsets = reinterpret_cast<int32_t*>(base + d.offsets_at);
    auto* tokens = reinterpret_cast<int32_t*>(base + d.tokens_at);
    int32_t cursor = 0;
    for (size_t i = 0; ok && i < plan.appends.size(); ++i) {
      const Append& a = plan.appends[i];
      slot_list[i] = a.slot;
      offsets[i] = cursor;
      ok = gather(a, vocab, tokens + cursor);
      cursor += (int32_t)a.count;
    }
    offsets[plan.appends.size()] = cursor;
  }
  if (!ok) {
    forget(book, plan);
    return nullptr;
  }
  const std::vector<int8_t>& logprobs = b->logprobs;
  const hs_row_out* rec = nullptr;
  Py_BEGIN_ALLOW_THREADS
  st = s->step(s->h, logits, dtype, stride, (int)n, vocab, &d, &rec, stream);
  Py_END_ALLOW_THREADS
  Ref out(st == HS_OK && !packed ? blank_samples(n, logprobs.data(), vocab) : nullptr);
  if (st == HS_OK) {
    Py_BEGIN_ALLOW_THREADS
    st = s->wait(s->h, stream);
    Py_END_ALLOW_THREADS
  }
  if (st != HS_OK) {
    PyErr_Clear();
    forget(book, plan);
    return failed(s, "hs_step", st);
  }
  if (!out && !packed) return nullptr;
  int status = 0;
  for (Py_ssize_t i = 0; i < n; ++i) status |= rec[i].status;
  // (rows without log-probabilities leave that part of the pinned record as it was)
  auto records = [&]() -> PyObject* {
    PyObject* copy = PyByteArray_FromStringAndSize(reinterpret_cast<const char*>(rec), n * (Py_ssize_t)sizeof(hs_row_out));
    auto* own = copy ? reinterpret_cast<hs_row_out*>(PyByteArray_AS_STRING(copy)) : nullptr;
    for (Py_ssize_t i = 0; own && i < n; ++i)
      if (own[i].n_top <= 0) {
        std::memset(own[i].top_ids, 0, sizeof own[i].top_ids);
        std::memset(own[i].top_logprobs, 0, sizeof own[i].top_logprobs);
      }
    return copy;
  };
  if (status & (2 | 4 | 64 | 128)) {
    Ref r(records());
    Ref p(PyByteArray_FromStringAndSize(reinterpret_cast<const char*>(rows), n * (Py_ssize_t)sizeof(hs_row_params)));
    if (!r || !p) return nullptr;
    return Py_BuildValue("[OO]", r.p, p.p);
  }
  if (packed) {
    Ref r(records());
    Ref l(PyBytes_FromStringAndSize(reinterpret_cast<const char*>(logprobs.data()), n));
    if (!r || !l) return nullptr;
    return Py_BuildValue("(OO)", r.p, l.p);
  }
  return filled_samples(out, rec, *b, vocab);
}

// greedy(logits address, dtype, row stride, batch, vocabulary, stream, packed) -> tuple of
// TokenSample, or (packed) the int32 token ids as a bytearray
PyObject* stepper_greedy(PyObject* self, PyObject* const* args, Py_ssize_t n_args) {
  auto* s = reinterpret_cast<Stepper*>(self);
  if (n_args != 7) {
    PyErr_SetString(PyExc_TypeError, "greedy takes seven arguments");
    return nullptr;
  }
  if (!s->h) return failed(s, "hs_step_greedy", HS_ERR_INVALID);
  const void* logits = reinterpret_cast<const void*>((uintptr_t)PyLong_AsUnsignedLongLong(args[0]));
  const int dtype = (int)PyLong_AsLong(args[1]);
  const int64_t stride = PyLong_AsLongLong(args[2]);
  const int n = (int)PyLong_AsLong(args[3]);
  const int vocab = (int)PyLong_AsLong(args[4]);
  void* stream = reinterpret_cast<void*>((uintptr_t)PyLong_AsUnsignedLongLong(args[5]));
  const int packed = PyObject_IsTrue(args[6]);
  if (PyErr_Occurred()) return nullptr;
  const int32_t* tokens = nullptr;
  int st;
  Py_BEGIN_ALLOW_THREADS
  st = s->greedy(s->h, logits, dtype, stride, n, vocab, &tokens, stream);
  Py_END_ALLOW_THREADS
  Ref out(st == HS_OK && !packed ? blank_samples(n, nullptr, vocab) : nullptr);
  if (st == HS_OK) {
    Py_BEGIN_ALLOW_THREADS
    st = s->wait(s->h, stream);
    Py_END_ALLOW_THREADS
  }
  if (st != HS_OK) {
    PyErr_Clear();
    return failed(s, "hs_step_greedy", st);
  }
  if (packed) return PyByteArray_FromStringAndSize(reinterpret_cast<const char*>(tokens), n * (Py_ssize_t)4);
  if (!out) return nullptr;
  for (int i = 0; i < n; ++i)
    if (!set_token(PyTuple_GET_ITEM(out.p, i), tokens[i])) return nullptr;
  return out.take();
}

PyMethodDef stepper_methods[] = {
    {"step", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(stepper_step)), METH_FASTCALL, "One sampling step."},
    {"greedy", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(stepper_greedy)), METH_FASTCALL, "One plain-greedy step."},
    {"close", stepper_close, METH_NOARGS, "The sampler is gone: steps fail from here on."},
    {nullptr, nullptr, 0, nullptr}};

// ---- module functions --------------------------------------------------------------------------------
// bind(TokenSample, as_int64, unseeded_keys)
PyObject* mod_bind(PyObject*, PyObject* args) {
  PyObject *type, *as_int64, *keys;
  if (!PyArg_ParseTuple(args, "OOO", &type, &as_int64, &keys)) return nullptr;
  const char* names[3] = {"token_id", "logprob", "top_logprobs"};
  Py_ssize_t* offsets[3] = {&g.off_token, &g.off_logprob, &g.off_top};
  for (int i = 0; i < 3; ++i) {
    Ref d(PyObject_GetAttrString(type, names[i]));
    if (!d) return nullptr;
    if (!Py_IS_TYPE(d.p, &PyMemberDescr_Type)) {
      PyErr_Format(PyExc_TypeError, "%s is not a slot", names[i]);
      return nullptr;
    }
    *offsets[i] = reinterpret_cast<PyMemberDescrObject*>(d.p)->d_member->offset;
  }
  Py_XSETREF(g.token_sample, Py_NewRef(type));
  Py_XSETREF(g.as_int64, Py_NewRef(as_int64));
  Py_XSETREF(g.unseeded_keys, Py_NewRef(keys));
  Py_RETURN_NONE;
}
// batch(params) -> (the params, packed static part, any unseeded row, seeds or None, which rows
// have penalties), the same object for the same parameter objects
PyObject* mod_batch(PyObject*, PyObject* params) {
  Ref t(PySequence_Tuple(params));
  if (!t) return nullptr;
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(t.p)->ob_item, PyTuple_GET_SIZE(t.p));
  return b ? Py_NewRef(b->view) : nullptr;
}
// traits(params) -> (lowest top_k, highest top_k, any row with temperature 0, any unseeded row, any
// row with penalties)
PyObject* mod_traits(PyObject*, PyObject* params) {
  Ref t(PySequence_Tuple(params));
  if (!t) return nullptr;
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(t.p)->ob_item, PyTuple_GET_SIZE(t.p));
  if (!b) return nullptr;
  return Py_BuildValue("(iiOOO)", b->top_k_lo, b->top_k_hi, b->any_zero_t ? Py_True : Py_False,
                       b->any_unseeded ? Py_True : Py_False, b->any_penalised ? Py_True : Py_False);
}
// survey(histories, params[, steps]) -> -1 when every row is plain greedy, else the longest history
// of a row with penalties.  Raises for a step that is no number (a plain greedy row has no use for its own).
PyObject* mod_survey(PyObject*, PyObject* const* args, Py_ssize_t n_args) {
  if (n_args != 2 && n_args != 3) {
    PyErr_SetString(PyExc_TypeError, "survey takes two or three arguments");
    return nullptr;
  }
  if (n_args == 3) {
    Ref steps(PySequence_Tuple(args[2]));
    if (!steps) return nullptr;
    for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(steps.p); ++i) {
      if (PyLong_CheckExact(PyTuple_GET_ITEM(steps.p, i))) continue;
      Ref number(PyNumber_Long(PyTuple_GET_ITEM(steps.p, i)));
      if (!number) return nullptr;
    }
  }
  Ref params(PySequence_Tuple(args[1])), histories(PySequence_Tuple(args[0]));
  if (!params || !histories) return nullptr;
  const Py_ssize_t n = PyTuple_GET_SIZE(params.p);
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(params.p)->ob_item, n);
  if (!b) return nullptr;
  if (b->all_greedy) return PyLong_FromLong(-1);
  long long longest = 0;
  if (b->any_penalised) {
    for (Py_ssize_t i = 0; i < n && i < PyTuple_GET_SIZE(histories.p); ++i) {
      if (!b->penalised[(size_t)i]) continue;
      const long long len = length(PyTuple_GET_ITEM(histories.p, i));
      if (len < 0) return nullptr;
      if (len > longest) longest = len;
    }
  }
  return PyLong_FromLongLong(longest);
}
// pack(params, steps, slots or None, unseeded keys or None) -> hs_row_params per row, a bytearray
PyObject* mod_pack(PyObject*, PyObject* args) {
  PyObject *params_in, *steps_in, *slots_in, *keys_in;
  if (!PyArg_ParseTuple(args, "OOOO", &params_in, &steps_in, &slots_in, &keys_in)) return nullptr;
  Ref params(PySequence_Tuple(params_in)), steps(PySequence_Tuple(steps_in));
  if (!params || !steps) return nullptr;
  Ref slots(slots_in == Py_None ? nullptr : PySequence_Tuple(slots_in));
  if (!slots && slots_in != Py_None) return nullptr;
  const Py_ssize_t n = PyTuple_GET_SIZE(params.p);
  if (PyTuple_GET_SIZE(steps.p) != n || (slots && PyTuple_GET_SIZE(slots.p) != n)) {
    PyErr_SetString(PyExc_ValueError, "one step and one slot per row");
    return nullptr;
  }
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(params.p)->ob_item, n);
  if (!b) return nullptr;
  Ref keys(nullptr);
  if (b->any_unseeded) {
    keys.p = keys_in == Py_None ? PyObject_CallOneArg(g.unseeded_keys, params.p) : Py_NewRef(keys_in);
    if (!keys) return nullptr;
  }
  Ref out(PyByteArray_FromStringAndSize(reinterpret_cast<const char*>(b->rows.data()), n * (Py_ssize_t)sizeof(hs_row_params)));
  if (!out) return nullptr;
  auto* rows = reinterpret_cast<hs_row_params*>(PyByteArray_AS_STRING(out.p));
  if (!mix_seeds(*b, reinterpret_cast<PyTupleObject*>(steps.p)->ob_item, keys.p, rows)) return nullptr;
  for (Py_ssize_t i = 0; slots && i < n; ++i) {
    const long v = PyLong_AsLong(PyTuple_GET_ITEM(slots.p, i));
    if (v == -1 && PyErr_Occurred()) return nullptr;
    rows[i].slot = (int32_t)v;
  }
  return out.take();
}
// plan(book, first per-call slot, histories, params, request ids or None) -> (slot per row,
// slots to reset, [(slot, tokens to append)])
PyObject* mod_plan(PyObject*, PyObject* args) {
  PyObject *book, *histories_in, *params_in, *ids_in;
  int base;
  if (!PyArg_ParseTuple(args, "O!iOOO", &SlotBookType, &book, &base, &histories_in, &params_in, &ids_in)) return nullptr;
  Ref histories(PySequence_Tuple(histories_in)), params(PySequence_Tuple(params_in));
  if (!histories || !params) return nullptr;
  Ref ids(ids_in == Py_None ? nullptr : PySequence_Tuple(ids_in));
  if (!ids && ids_in != Py_None) return nullptr;
  const Py_ssize_t n = PyTuple_GET_SIZE(params.p);
  if (PyTuple_GET_SIZE(histories.p) != n || (ids && PyTuple_GET_SIZE(ids.p) != n)) {
    PyErr_SetString(PyExc_ValueError, "sampling metadata must match the logits batch");
    return nullptr;
  }
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(params.p)->ob_item, n);
  if (!b) return nullptr;
  StepPlan plan;
  std::vector<int> slots((size_t)n, -1);
  auto undo = [&]() -> PyObject* {
    forget(reinterpret_cast<SlotBook*>(book), plan);
    return nullptr;
  };
  if (!plan_step(reinterpret_cast<SlotBook*>(book), base, *b, reinterpret_cast<PyTupleObject*>(histories.p)->ob_item,
                 ids ? ids.p : nullptr, slots.data(), plan))
    return undo();
  Ref out_slots(PyList_New(0)), resets(PyList_New(0)), appends(PyList_New(0));
  if (!out_slots || !resets || !appends) return undo();
  auto push = [](PyObject* list, PyObject* o) {
    const bool ok = o && PyList_Append(list, o) == 0;
    Py_XDECREF(o);
    return ok;
  };
  for (int v : slots)
    if (!push(out_slots.p, PyLong_FromLong(v))) return undo();
  for (int v : plan.resets)
    if (!push(resets.p, PyLong_FromLong(v))) return undo();
  for (const Append& a : plan.appends) {
    PyObject* tail = tail_of(a);
    if (!tail) return undo();
    if (!push(appends.p, Py_BuildValue("(iN)", a.slot, tail))) return undo();
  }
  return PyTuple_Pack(3, out_slots.p, resets.p, appends.p);
}
// Samples without their numbers, made while the GPU is at work (for a caller that does not use a Stepper).
// They stay in a capsule until there are records to fill them from: nobody sees them half made.  (Calls of 32
// to 512 rows with 20 log-probabilities take 5 to 14 % less than with objects made after the records; to stop at
// some number of them is slower at every size from 192 rows on: 256 rows of 128,000 374 us, with 2,688 objects
// at most 404.)
struct Blank {
  PyObject* samples;
  std::vector<int8_t> logprobs;
  int vocab;
};
constexpr const char* kBlank = "hydraserve_b200._host.blank";
void blank_free(PyObject* capsule) {
  auto* b = static_cast<Blank*>(PyCapsule_GetPointer(capsule, kBlank));
  if (!b) return;
  Py_XDECREF(b->samples);
  delete b;
}
// blank(params, vocab) -> a capsule for samples()
PyObject* mod_blank(PyObject*, PyObject* args) {
  PyObject* params_in;
  int vocab;
  if (!PyArg_ParseTuple(args, "Oi", &params_in, &vocab)) return nullptr;
  Ref params(PySequence_Tuple(params_in));
  if (!params) return nullptr;
  const Py_ssize_t n = PyTuple_GET_SIZE(params.p);
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(params.p)->ob_item, n);
  if (!b) return nullptr;
  Ref made(blank_samples(n, b->logprobs.data(), vocab));
  if (!made) return nullptr;
  auto* blank = new Blank{made.take(), b->logprobs, vocab};
  PyObject* capsule = PyCapsule_New(blank, kBlank, blank_free);
  if (!capsule) {
    Py_DECREF(blank->samples);
    delete blank;
  }
  return capsule;
}
// samples(records, params, vocab[, blank]) -> the samples, the blank ones (which are used up) if they are of this batch
PyObject* mod_samples(PyObject*, PyObject* args) {
  PyObject *records, *params_in, *capsule = Py_None;
  int vocab;
  if (!PyArg_ParseTuple(args, "OOi|O", &records, &params_in, &vocab, &capsule)) return nullptr;
  Ref params(PySequence_Tuple(params_in));
  if (!params) return nullptr;
  const Py_ssize_t n = PyTuple_GET_SIZE(params.p);
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(params.p)->ob_item, n);
  if (!b) return nullptr;
  Py_buffer view;
  if (PyObject_GetBuffer(records, &view, PyBUF_C_CONTIGUOUS) < 0) return nullptr;
  PyObject* out = nullptr;
  if (view.len != n * (Py_ssize_t)sizeof(hs_row_out)) PyErr_SetString(PyExc_ValueError, "one record per row");
  else {
    const auto* rec = static_cast<const hs_row_out*>(view.buf);
    auto* blank = capsule == Py_None ? nullptr : static_cast<Blank*>(PyCapsule_GetPointer(capsule, kBlank));
    if (blank && blank->samples && blank->vocab == vocab && blank->logprobs == b->logprobs) {
      Ref made(blank->samples);
      blank->samples = nullptr;
      out = filled_samples(made, rec, *b, vocab);
    } else if (!PyErr_Occurred()) {
      out = samples_of(rec, *b, vocab);
    }
  }
  PyBuffer_Release(&view);
  return out;
}
// logprob_codes(params) -> int8 per row: log-probabilities asked for, -1 = none
PyObject* mod_codes(PyObject*, PyObject* params) {
  Ref t(PySequence_Tuple(params));
  if (!t) return nullptr;
  const BatchRef b = batch_of(reinterpret_cast<PyTupleObject*>(t.p)->ob_item, PyTuple_GET_SIZE(t.p));
  return b ? PyBytes_FromStringAndSize(reinterpret_cast<const char*>(b->logprobs.data()), (Py_ssize_t)b->logprobs.size()) : nullptr;
}

// batched_greedy() -> False when HYDRASERVE_BATCHED_GREEDY is "0" (os.environ's writes reach the C
// environment; reading it through os.environ costs a microsecond per call)
PyObject* mod_batched_greedy(PyObject*, PyObject*) {
  const char* v = std::getenv("HYDRASERVE_BATCHED_GREEDY");
  return PyBool_FromLong(!(v && v[0] == '0' && v[1] == 0));
}

PyMethodDef module_methods[] = {
    {"batched_greedy", mod_batched_greedy, METH_NOARGS, "Whether the batched arg-max path is on."},
    {"bind", mod_bind, METH_VARARGS, "Hand over the Python objects this module works with."},
    {"batch", mod_batch, METH_O, "What depends on a batch's parameters alone."},
    {"traits", mod_traits, METH_O, "What a vocabulary-sharded call asks about a batch's parameters."},
    {"survey", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(mod_survey)), METH_FASTCALL, "-1 for an all plain-greedy batch, else the longest penalised history."},
    {"pack", mod_pack, METH_VARARGS, "hs_row_params of a batch."},
    {"plan", mod_plan, METH_VARARGS, "Histogram slots of a batch."},
    {"blank", mod_blank, METH_VARARGS, "Samples without their numbers, for samples()."},
    {"samples", mod_samples, METH_VARARGS, "Records to TokenSample objects."},
    {"logprob_codes", mod_codes, METH_O, "Log-probabilities asked for per row."},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host", "Host side of a sampling step.", -1, module_methods,
                          nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
  entry_seq.sq_length = entry_len;
  entry_seq.sq_item = entry_item;
  entry_seq.sq_ass_item = entry_set;
  SlotEntryType.tp_name = "hydraserve_b200._host.SlotEntry";
  SlotEntryType.tp_basicsize = sizeof(SlotEntry);
  SlotEntryType.tp_dealloc = entry_dealloc;
  SlotEntryType.tp_as_sequence = &entry_seq;
  SlotEntryType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
  SlotEntryType.tp_traverse = entry_traverse;
  SlotEntryType.tp_doc = "(slot, tokens counted) of one request";
  SlotBookType.tp_name = "hydraserve_b200._host.SlotBook";
  SlotBookType.tp_basicsize = sizeof(SlotBook);
  SlotBookType.tp_dealloc = book_dealloc;
  SlotBookType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
  SlotBookType.tp_traverse = book_traverse;
  SlotBookType.tp_clear = book_clear;
  SlotBookType.tp_doc = "Which request holds which resident histogram slot, and how much of its history the "
                        "device has counted; least recently used requests are evicted first, never one of the batch.";
  SlotBookType.tp_methods = book_methods;
  SlotBookType.tp_members = book_members;
  SlotBookType.tp_new = book_new;
  SlotBookType.tp_init = book_init;
  StepperType.tp_name = "hydraserve_b200._host.Stepper";
  StepperType.tp_basicsize = sizeof(Stepper);
  StepperType.tp_dealloc = stepper_dealloc;
  StepperType.tp_flags = Py_TPFLAGS_DEFAULT | Py_TPFLAGS_HAVE_GC;
  StepperType.tp_traverse = stepper_traverse;
  StepperType.tp_doc = "Runs the steps of one sampler.";
  StepperType.tp_methods = stepper_methods;
  StepperType.tp_new = stepper_new;
  if (PyType_Ready(&SlotEntryType) < 0 || PyType_Ready(&SlotBookType) < 0 || PyType_Ready(&StepperType) < 0) return nullptr;
  struct { PyObject** at; const char* name; } names[] = {
      {&s_temperature, "temperature"}, {&s_top_p, "top_p"}, {&s_top_k, "top_k"}, {&s_min_p, "min_p"},
      {&s_repetition, "repetition_penalty"}, {&s_presence, "presence_penalty"}, {&s_frequency, "frequency_penalty"},
      {&s_seed, "seed"}, {&s_logprobs, "logprobs"}};
  for (auto& e : names)
    if (!(*e.at = PyUnicode_InternFromString(e.name))) return nullptr;
  g.neg_inf = PyFloat_FromDouble(-Py_HUGE_VAL);
  g.empty = PyTuple_New(0);
  PyObject* m = PyModule_Create(&module_def);
  if (!m || !g.neg_inf || !g.empty) return nullptr;
  if (PyModule_AddObjectRef(m, "SlotBook", reinterpret_cast<PyObject*>(&SlotBookType)) < 0 ||
      PyModule_AddObjectRef(m, "Stepper", reinterpret_cast<PyObject*>(&StepperType)) < 0)
    return nullptr;
  return m;
}
